"""The staged mode's gate kernel with a launch per layer (few words, many gates):
against the oracle at the edges of its tiles, of one and of many separate trees,
and on both sides of the line between the two ways."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200.graph import AND, ATLEAST, NAND, NOR, OR, XOR, probability_threshold


def _layered(n_be, n_gates, layers, fan, n_small=0, seed=0, kinds=(AND, OR, NAND, NOR, XOR, ATLEAST)):
    """Gates in equal layers, each reading the layer below, under one top; and n_small trees of one gate and two
    events of their own beside them."""
    rng = np.random.default_rng(seed)
    per = (n_gates - 1) // layers
    nb = n_be + 2 * n_small
    ops, ks, count, neg, inputs = [], [], [], [], []

    def gate(op, inp, negated):
        ops.append(op)
        ks.append(max(1, len(inp) // 2))
        count.append(len(inp))
        neg.append(negated)
        inputs.extend(int(x) for x in inp)

    for level in range(layers):
        lo, hi = (0, n_be) if level == 0 else (nb + (level - 1) * per, nb + level * per)
        for _ in range(per):
            gate(int(rng.choice(kinds)), rng.integers(lo, hi, fan), int(rng.integers(0, fan + 1)))
    gate(OR, range(nb + (layers - 1) * per, nb + layers * per), 0)
    for t in range(n_small):
        gate(XOR, [n_be + 2 * t, n_be + 2 * t + 1], 1)
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + nb), be_event_idx=rng.permutation(nb),
                       be_threshold=probability_threshold(rng.uniform(0.05, 0.95, nb)), gate_op=ops, gate_k=ks,
                       gate_in_begin=np.concatenate([[0], np.cumsum(count)[:-1]]), gate_in_count=count,
                       gate_neg_count=neg, inputs=inputs, tally_nodes=np.arange(nb, nb + len(ops)))


def _run(capi, g, words, chunk=0, begin=3):
    with capi.Engine(g, mode=capi.MODE_STAGED, layered_max_words=chunk) as e:
        e.run(2, 1, begin, words)
        ones, total = e.tallies()
        launches = e.launch_count()
    assert total == words * 64
    return ones, launches


@pytest.mark.gpu
@pytest.mark.parametrize("n_small", [0, 3, 90])
@pytest.mark.parametrize("words,chunk", [(1, 0), (31, 0), (32, 0), (33, 0), (100, 0), (700, 256), (1025, 0)])
def test_layers_in_launches_of_their_own(capi, oracle_mod, gpu, words, chunk, n_small):
    g = _layered(60, 2401, 3, 5, n_small)
    ones, launches = _run(capi, g, words, chunk)
    assert np.array_equal(ones, oracle_mod.tallies(g, 2, 1, 3, words))
    chunks = -(-words // (chunk or words))
    assert launches == 1 + 5 * chunks  # event table, then sampling and four layers


@pytest.mark.gpu
@pytest.mark.parametrize("fan,n_gates,layers,words,split", [(5, 2401, 3, 1025, True), (5, 2401, 3, 3000, False),
                                                            (5, 241, 30, 64, False), (60, 601, 4, 64, True),
                                                            (2, 121, 1, 64, False)])
def test_both_sides_of_the_line(capi, oracle_mod, gpu, fan, n_gates, layers, words, split):
    kinds = (ATLEAST,) if fan == 60 else (AND, OR)
    g = _layered(50, n_gates, layers, fan, kinds=kinds)
    ones, launches = _run(capi, g, words)
    assert np.array_equal(ones, oracle_mod.tallies(g, 2, 1, 3, words))
    assert launches == 2 + (layers + 1 if split else 1)
