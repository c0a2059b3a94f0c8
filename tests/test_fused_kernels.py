"""The fused mode's choice between the tile kernel and the interpreter: deep
graphs of few events, whose layers are a barrier each, go to the interpreter
where the words are many, and both give the oracle's tallies."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, OR, probability_threshold


def _deep(events, width, layers, fan=2, seed=0):
    """`width` chains of `layers` gates that each read the gate before and events, under one OR."""
    rng = np.random.default_rng(seed)
    inputs, count = [], []
    for level in range(layers):
        for k in range(width):
            below = [events + (level - 1) * width + k] if level else []
            inputs += below + [int(x) for x in rng.integers(0, events, fan - len(below))]
            count.append(fan)
    inputs += [events + (layers - 1) * width + k for k in range(width)]
    count.append(width)
    n = width * layers + 1
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + events), be_event_idx=np.arange(events),
                       be_threshold=probability_threshold(rng.uniform(0.05, 0.9, events)),
                       gate_op=[int(x) for x in rng.choice([AND, OR], n - 1)] + [OR], gate_k=np.zeros(n),
                       gate_in_begin=np.concatenate([[0], np.cumsum(count)[:-1]]), gate_in_count=count,
                       gate_neg_count=np.zeros(n), inputs=inputs, tally_nodes=[events + n - 1])


@pytest.mark.gpu
@pytest.mark.parametrize("events,width,layers,words,tile", [
    (60, 1, 800, 2048, True), (60, 1, 800, 70001, False), (20, 1, 200, 262144, False), (20, 1, 200, 4097, True),
    (500, 1, 800, 70001, False), (1000, 4, 800, 70001, False), (200, 16, 20, 70001, True)])
def test_deep_graphs(capi, oracle_mod, gpu, events, width, layers, words, tile):
    g = _deep(events, width, layers)
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        assert (e.fused_kernel(words)[0] > 0) == tile
        e.run(3, 2, 7, words)
        ones, total = e.tallies()
    assert total == 2 * words * 64
    assert np.array_equal(ones, oracle_mod.tallies(g, 3, 2, 7, words))


@pytest.mark.gpu
def test_trees_as_they_are_stay_with_the_tile_kernel(capi, gpu):
    for g in (synth.config1(), synth.small_tree(4)):
        with capi.Engine(g, mode=capi.MODE_FUSED) as e:
            assert all(e.fused_kernel(w)[0] > 0 for w in (1, 4096, 1 << 18, 1 << 32))
    with capi.Engine(synth.config1(), mode=capi.MODE_STRIP) as e:
        with pytest.raises(capi.McgError):
            e.fused_kernel(1)


def _read_through(events, gates, seed, share=0.2):
    """A tree whose top reaches every gate, so that its segments are all walked."""
    g = synth.generate(synth.TreeSpec(n_be=events, n_gates=gates, mix={AND: 0.5, OR: 0.5}, p_range=(0.1, 0.6), seed=seed,
                                      share_be_frac=share))
    return g.with_tallies([g.root, g.n_be + 1, 3, g.root])


@pytest.mark.gpu
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("threads", [256, 512])
def test_each_block_size_with_several_tiles_a_block(capi, oracle_mod, gpu, threads, side):
    """Trees whose rows leave room for four and for two blocks per SM, in the longest pass that takes larger blocks
    and in the shortest that does not."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = _read_through(*((130, 70) if threads == 256 else (250, 140)), seed=5)
    line = sms * (1024 // threads) * 32
    words = line - 32 if side == 0 else line + 45
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        assert e.fused_kernel(words) == (threads if side else 2 * threads, 1)
        assert e.fused_kernel(3 * line)[0] == threads
        for begin, n in ((5, words), (0, 3 * line - 7)):
            e.reset_tallies()
            e.run(2, 1, begin, n)
            assert np.array_equal(e.tallies()[0], oracle_mod.tallies(g, 2, 1, begin, n))


@pytest.mark.gpu
@pytest.mark.parametrize("events,gates,segments", [(600, 340, 2), (1030, 560, 4), (3000, 1700, 10)])
def test_tile_kernel_in_segments(capi, oracle_mod, gpu, events, gates, segments):
    g = _read_through(events, gates, seed=6)
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        for words in (33, 20011):
            threads, parts = e.fused_kernel(words)
            assert threads > 0 and parts >= segments
            e.reset_tallies()
            e.run(4, 2, 3, words)
            assert np.array_equal(e.tallies()[0], oracle_mod.tallies(g, 4, 2, 3, words))


@pytest.mark.gpu
def test_a_tree_that_does_not_fit(capi, oracle_mod, gpu):
    """Every event tallied keeps its row to the end: 1,600 rows are more than an SM holds."""
    g = _read_through(1600, 900, seed=7)
    g = g.with_tallies(np.arange(g.n_nodes))
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        assert e.fused_kernel(1000) == (0, 0)
        e.run(1, 1, 0, 1000)
        assert np.array_equal(e.tallies()[0], oracle_mod.tallies(g, 1, 1, 0, 1000))


@pytest.mark.gpu
def test_strip_and_batch_in_ten_segments_and_more(capi, oracle_mod, gpu):
    """5,000 events are 14 strip segments of 384, 1,200 are 12 batch segments of 96."""
    from mcscram_b200.uncertainty import Batch
    g = _read_through(5000, 2900, seed=8)
    with capi.Engine(g, mode=capi.MODE_STRIP) as e:
        e.run(3, 1, 11, 700)
        assert np.array_equal(e.tallies()[0], oracle_mod.tallies(g, 3, 1, 11, 700))
    t = _read_through(1200, 700, seed=9)
    rng = np.random.default_rng(9)
    thr = [probability_threshold(rng.uniform(0.05, 0.6, t.n_be)) for _ in range(5)]
    with Batch([t]) as b:
        got = b.run([0] * 5, thr, iteration=2, words_per_instance=70)
    for x, o in zip(thr, got):
        assert int(o) == int(np.sum(oracle_mod.tallies(t.with_thresholds(x), 2, 1, 0, 70)))
