"""The staged mode's gate kernel against the oracle: one and two words per lane,
odd and even row lengths, every connective with negated tails, wide gates and
every k of k-of-n gates, several chunks, and graphs of many separate trees."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200.graph import AND, ATLEAST, NAND, NOR, NOT, NULL, OR, XOR


def _trees(rng, n_trees, n_be, n_gates, fan_in, all_k=False):
    """n_trees separate graphs of n_be events and n_gates gates each, the gates in rounds over the trees."""
    ops, ks, begin, count, neg, inputs = [], [], [], [], [], []
    nb = n_trees * n_be
    for j in range(n_gates):
        for t in range(n_trees):
            op = ATLEAST if all_k else int(rng.choice([AND, OR, ATLEAST, XOR, NOT, NAND, NOR, NULL]))
            n = int(rng.choice(fan_in)) if j else 3
            pool = [t * n_be + i for i in range(n_be)] + [nb + i * n_trees + t for i in range(j)]
            ops.append(op)
            ks.append(j % (n + 2) if all_k else int(rng.integers(0, n + 2)))
            begin.append(len(inputs))
            count.append(n)
            neg.append(int(rng.integers(0, n + 1)))
            inputs += [int(x) for x in rng.choice(pool, n)]
    thr = rng.integers(1, 1 << 32, nb).astype(np.uint64)
    thr[0], thr[1] = 0, 1 << 32
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + nb), be_event_idx=rng.permutation(nb), be_threshold=thr,
                       gate_op=ops, gate_k=ks, gate_in_begin=begin, gate_in_count=count, gate_neg_count=neg,
                       inputs=inputs, tally_nodes=np.arange(nb + n_trees * n_gates))


def _check(capi, oracle_mod, g, words, begin=0, chunk=0, passes=1):
    with capi.Engine(g, mode=capi.MODE_STAGED, layered_max_words=chunk) as e:
        e.run(3, passes, begin, words)
        ones, total = e.tallies()
    want = sum(np.bitwise_count(oracle_mod.eval_words(g, 3 + i, begin, words)[g.tally_nodes]).sum(
        axis=1, dtype=np.uint64) for i in range(passes))
    assert total == passes * words * 64
    assert np.array_equal(ones, want)


@pytest.mark.gpu
@pytest.mark.parametrize("words,chunk,passes", [(1, 0, 1), (31, 0, 2), (64, 0, 1), (65, 0, 1), (1000, 256, 2),
                                                (9471, 0, 1), (9472, 0, 1), (9473, 0, 1), (9535, 0, 1),
                                                (40001, 9728, 1), (20000, 0, 1)])
def test_words(capi, oracle_mod, gpu, words, chunk, passes):
    rng = np.random.default_rng(words)
    g = _trees(rng, 1, 30, 40, [0, 1, 2, 3, 4, 5, 8, 9, 33])
    _check(capi, oracle_mod, g, words, begin=7, chunk=chunk, passes=passes)


@pytest.mark.gpu
@pytest.mark.parametrize("fan_in", [[2], [4], [7], [8], [12], [256, 300]])
def test_every_k(capi, oracle_mod, gpu, fan_in):
    rng = np.random.default_rng(fan_in[0])
    g = _trees(rng, 1, 20, 30, fan_in, all_k=True)
    for words in (33, 9600):
        _check(capi, oracle_mod, g, words)


@pytest.mark.gpu
@pytest.mark.parametrize("n_trees", [2, 64, 65, 150])
def test_separate_trees(capi, oracle_mod, gpu, n_trees):
    rng = np.random.default_rng(n_trees)
    g = _trees(rng, n_trees, 6, 9, [1, 2, 3, 6])
    for words, chunk in ((100, 0), (9601, 0), (700, 256)):
        _check(capi, oracle_mod, g, words, chunk=chunk)


@pytest.mark.gpu
def test_events_only(capi, oracle_mod, gpu):
    g = G.FlatGraph(be_pdag_idx=[2, 3], be_event_idx=[0, 1], be_threshold=[1 << 31, 1 << 30], gate_op=[], gate_k=[],
                    gate_in_begin=[], gate_in_count=[], gate_neg_count=[], inputs=[], tally_nodes=[0, 1])
    _check(capi, oracle_mod, g, 77)
