"""The choice between the batch tile kernel and the interpreter: few instances of
deep trees on many words go to the interpreter, and one handle may take both in
turn, with the oracle's counts from either."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, OR, probability_threshold


def _chain(events, gates, seed=0):
    """Gate j reads gate j - 1 and an event."""
    rng = np.random.default_rng(seed)
    inputs = [x for j in range(gates) for x in ([events + j - 1] if j else [0]) + [int(rng.integers(0, events))]]
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + events), be_event_idx=np.arange(events),
                       be_threshold=probability_threshold(rng.uniform(0.05, 0.9, events)),
                       gate_op=[int(x) for x in rng.choice([AND, OR], gates)], gate_k=np.zeros(gates),
                       gate_in_begin=2 * np.arange(gates), gate_in_count=np.full(gates, 2),
                       gate_neg_count=np.zeros(gates), inputs=inputs, tally_nodes=[events + gates - 1])


@pytest.mark.gpu
def test_one_handle_takes_both_in_turn(oracle_mod, gpu):
    from mcscram_b200.uncertainty import Batch
    c1 = synth.config1()
    trees = [_chain(60, 400), c1.with_tallies([c1.root])]
    rng = np.random.default_rng(3)
    thr = [[probability_threshold(rng.uniform(0.05, 0.8, t.n_be)) for _ in range(17)] for t in trees]
    runs = [([0], 1 << 17, False), ([0], 1024, True), ([1] * 16, 1 << 15, True), ([0, 0], 100001, False),
            ([1] * 17, 2048, True), ([0] * 5 + [1] * 2, 90000, False), ([0], 1 << 17, False)]
    with Batch(trees) as b:
        for inst, words, tiles in runs:
            assert b.takes_tiles(inst, words) == tiles, (inst, words)
            seen = [0, 0]
            use = []
            for t in inst:
                use.append(thr[t][seen[t]])
                seen[t] += 1
            got = b.run(inst, use, iteration=2, words_per_instance=words)
            for t, th, o in zip(inst, use, got):
                assert int(o) == int(oracle_mod.tallies(trees[t].with_thresholds(th), 2, 1, 0, words)[0])


@pytest.mark.gpu
def test_draws_of_ordinary_trees_stay_with_the_tile_kernel(gpu):
    from mcscram_b200.uncertainty import Batch
    c1, c2 = synth.config1(), synth.config2()
    with Batch([c1.with_tallies([c1.root]), c2.with_tallies([c2.root])]) as b:
        for tree in (0, 1):
            for n in (1, 4, 16, 101):
                assert all(b.takes_tiles([tree] * n, w) for w in (64, 4096, 1 << 16))
    with Batch([c1.with_tallies([c1.root])], ctas_per_sm=4) as b:  # a launch shape of its own is the interpreter's
        assert not b.takes_tiles([0] * 16, 4096)
