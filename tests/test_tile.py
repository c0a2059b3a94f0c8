"""The fused mode's tile kernel (trees whose node words fit in shared memory)
against the oracle: tile and block edges of a pass, every connective with
negated tails, constant events, single-event and event-only tallies, trees at
each block size, and the first size that no longer fits."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, ATLEAST, NAND, NOR, NOT, NULL, OR, XOR


def _every_connective(rng, n_be=40, n_gates=60):
    """Random gates of all connectives with negated tails, empty gates, wide
    gates and shared inputs; thresholds 0 and 2^32 among the events."""
    ops, ks, begin, count, neg, inputs = [], [], [], [], [], []
    for j in range(n_gates):
        op = int(rng.choice([AND, OR, ATLEAST, XOR, NOT, NAND, NOR, NULL]))
        n = int(rng.choice([0, 1, 2, 3, 5, 9, 16, 33])) if j else 3
        ops.append(op)
        ks.append(int(rng.integers(0, n + 2)))
        begin.append(len(inputs))
        count.append(n)
        neg.append(int(rng.integers(0, n + 1)))
        inputs += [int(x) for x in rng.integers(0, n_be + j, n)]
    thr = rng.integers(1, 1 << 32, n_be).astype(np.uint64)
    thr[0], thr[1] = 0, 1 << 32
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n_be), be_event_idx=rng.permutation(n_be), be_threshold=thr,
                       gate_op=ops, gate_k=ks, gate_in_begin=begin, gate_in_count=count, gate_neg_count=neg,
                       inputs=inputs, tally_nodes=np.arange(n_be + n_gates))


def _popcounts(words):
    return np.array([int(np.unpackbits(r.view(np.uint8)).sum()) for r in words], dtype=np.uint64)


def _check(capi, oracle_mod, g, words, begin=0, passes=1, first=1):
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        e.run(first, passes, begin, words)
        ones, total = e.tallies()
    want = sum(_popcounts(oracle_mod.eval_words(g, first + i, begin, words)[g.tally_nodes]) for i in range(passes))
    assert total == passes * words * 64
    assert np.array_equal(ones, want)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(4))
def test_every_connective(capi, oracle_mod, gpu, seed):
    _check(capi, oracle_mod, _every_connective(np.random.default_rng(seed)), 45, passes=2)


@pytest.mark.gpu
@pytest.mark.parametrize("words,begin", [(1, 0), (31, 5), (32, 0), (33, 7), (1000, 123), (20000, 0),
                                         (40, (1 << 32) - 40)])
def test_pass_edges(capi, oracle_mod, gpu, words, begin):
    g = synth.config1()
    _check(capi, oracle_mod, g.with_tallies(np.arange(g.n_nodes)), words, begin, passes=1 if words > 5000 else 3, first=7)


@pytest.mark.gpu
@pytest.mark.parametrize("n_be,n_gates", [(6, 3), (130, 70), (160, 80), (280, 150), (560, 300), (620, 320)])
def test_block_sizes_and_the_first_tree_that_does_not_fit(capi, oracle_mod, gpu, n_be, n_gates):
    # 56 KB, 113 KB and 227 KB of words (4, 2 and 1 blocks an SM), and past them
    g = synth.generate(synth.TreeSpec(n_be=n_be, n_gates=n_gates, mix={AND: 0.5, OR: 0.5}, p_range=(0.05, 0.5),
                                      seed=5, share_be_frac=0.2))
    _check(capi, oracle_mod, g.with_tallies(np.arange(n_be, g.n_nodes)), 333)


@pytest.mark.gpu
def test_event_tallies_without_gates_and_repeated_nodes(capi, oracle_mod, gpu):
    g = synth.config1()
    _check(capi, oracle_mod, g.with_tallies([3, 5, 3, 199]), 70)
    _check(capi, oracle_mod, g.with_tallies([g.root, 4, g.root, g.n_be + 10]), 70)
    _check(capi, oracle_mod, g.with_tallies(list(range(g.n_nodes)) * 40), 70)  # more counters than shared memory holds


@pytest.mark.gpu
@pytest.mark.parametrize("draws,words", [((1,), 1), ((4, 5), 31), ((8, 9), 32), ((16,), 33), ((17, 3), 64),
                                         ((33, 1, 16), 100), ((2, 15), 2049)])
def test_batched_instances_in_tiles(oracle_mod, gpu, draws, words):
    """Group sizes around the kernel's 4, 8 and 16 thresholds at a time, passes
    around a tile, every connective, wide ATLEAST gates, constant thresholds
    inside a group, rare and near-certain events, tallied events and nodes
    tallied twice: every instance equals the oracle at its own thresholds."""
    from mcscram_b200.uncertainty import Batch
    rng = np.random.default_rng(len(draws) * 1000 + words)
    trees = [synth.config1().with_tallies([299]), _every_connective(np.random.default_rng(1)),
             synth.small_tree(4).with_tallies([35, 2, 35, 2, 30])]
    inst_tree, thr = [], []
    for t, n in enumerate(draws):
        for d in range(n):
            p = 10.0 ** rng.uniform(-4, 0, trees[t].n_be) if d % 3 else rng.uniform(0.5, 1.0, trees[t].n_be)
            th = np.minimum((p * 2.0**32).astype(np.uint64), np.uint64((1 << 32) - 1))
            if d % 4 == 1:
                th[:3] = [0, 1 << 32, (1 << 32) - 1]
            if d % 5 == 4:
                th[:] = np.where(rng.random(th.size) < 0.5, 0, 1 << 32)
            inst_tree.append(t)
            thr.append(th)
    order = rng.permutation(len(inst_tree))  # runs of one tree, and groups of one
    runs = list(range(len(inst_tree))) + [int(i) for i in order]
    with Batch(trees) as b:
        got = b.run([inst_tree[i] for i in runs], [thr[i] for i in runs], iteration=5, words_per_instance=words)
    for i, o in zip(runs, got):
        g = trees[inst_tree[i]].with_thresholds(thr[i])
        assert int(o) == int(np.sum(oracle_mod.tallies(g, 5, 1, 0, words))), (i, inst_tree[i])


def _far_reads(rng, n_be, n_gates, tallies):
    """Gates that read the last 40 gates and any event up to their share of them."""
    ops, ks, begin, count, neg, inputs = [], [], [], [], [], []
    for j in range(n_gates):
        op = int(rng.choice([AND, OR, ATLEAST, XOR, NOT, NAND, NOR, NULL]))
        n = 1 if op in (NOT, NULL) else int(rng.integers(2, 7))
        last = max(1, min(n_be, (j + 1) * n_be // n_gates))
        pool = np.concatenate([rng.integers(0, last, n), n_be + rng.integers(max(0, j - 40), j, n)]) if j else \
            rng.integers(0, last, n)
        ops.append(op)
        ks.append(int(rng.integers(1, n + 1)))
        begin.append(len(inputs))
        count.append(n)
        neg.append(int(rng.integers(0, n + 1)))
        inputs += [int(x) for x in rng.choice(pool, n)]
    nodes = n_be + n_gates
    tally = {"root": [nodes - 1], "all": np.arange(nodes), "some": rng.integers(0, nodes, 25)}[tallies]
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n_be), be_event_idx=rng.permutation(n_be),
                       be_threshold=(10.0 ** rng.uniform(-3, 0, n_be) * 2.0**32).astype(np.uint64), gate_op=ops,
                       gate_k=ks, gate_in_begin=begin, gate_in_count=count, gate_neg_count=neg, inputs=inputs,
                       tally_nodes=tally)


@pytest.mark.gpu
@pytest.mark.parametrize("n_be,n_gates,tallies", [(95, 60, "root"), (96, 60, "all"), (700, 420, "root"),
                                                  (700, 420, "some"), (1200, 700, "all"), (250, 0, "all")])
def test_batched_trees_in_segments(oracle_mod, gpu, n_be, n_gates, tallies):
    """Trees of several segments, whose rows are used again: nodes read far from
    where they are written, tallied events (their rows last), events no gate reads."""
    from mcscram_b200.uncertainty import Batch
    rng = np.random.default_rng(n_be + n_gates)
    g = _far_reads(rng, n_be, n_gates, tallies)
    thr = [(10.0 ** rng.uniform(-3, 0, n_be) * 2.0**32).astype(np.uint64) for _ in range(6)]
    with Batch([g]) as b:
        got = b.run([0] * len(thr), thr, iteration=2, words_per_instance=70)
    for t, o in zip(thr, got):
        assert int(o) == int(np.sum(oracle_mod.tallies(g.with_thresholds(t), 2, 1, 0, 70)))


@pytest.mark.gpu
@pytest.mark.parametrize("n_be,n_gates,tallies", [(383, 200, "all"), (385, 300, "some"), (1600, 1000, "all"),
                                                  (1600, 1000, "root"), (900, 0, "all")])
def test_strip_segments(capi, oracle_mod, gpu, n_be, n_gates, tallies):
    """The strip mode's segments and reused rows on the same graphs, and on one of
    every connective with empty and wide gates."""
    g = _far_reads(np.random.default_rng(n_be + n_gates), n_be, n_gates, tallies)
    for h in (g, _every_connective(np.random.default_rng(n_be))):
        with capi.Engine(h, mode=capi.MODE_STRIP) as e:
            e.run(4, 2, 3, 300)
            ones, total = e.tallies()
        want = sum(_popcounts(oracle_mod.eval_words(h, 4 + i, 3, 300)[h.tally_nodes]) for i in range(2))
        assert total == 2 * 300 * 64
        assert np.array_equal(ones, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n_be,n_gates,tallies,words", [(600, 400, "all", 40), (900, 700, "root", 33),
                                                        (1600, 1000, "some", 64), (1600, 1000, "all", 5000),
                                                        (3000, 300, "root", 100), (900, 0, "all", 70)])
def test_tile_segments(capi, oracle_mod, gpu, n_be, n_gates, tallies, words):
    """The fused mode's default shape on trees beyond the tile: in segments, or by
    the interpreter where too many nodes are live at a time."""
    g = _far_reads(np.random.default_rng(n_be * 3 + n_gates), n_be, n_gates, tallies)
    _check(capi, oracle_mod, g, words, 9, passes=2)


@pytest.mark.gpu
@pytest.mark.parametrize("words", [1, 256, 257, 4 * 148 * 256, 4 * 148 * 256 + 1])
def test_strip_grid(capi, oracle_mod, gpu, words):
    """Strip passes of fewer strips than blocks, and both sides of the line between the kernels."""
    g = synth.small_tree(4)
    g = g.with_tallies(np.arange(g.n_nodes))
    with capi.Engine(g, mode=capi.MODE_STRIP) as e:
        e.run(2, 1, 11, words)
        ones, total = e.tallies()
    assert total == words * 64
    assert np.array_equal(ones, _popcounts(oracle_mod.eval_words(g, 2, 11, words)[g.tally_nodes]))
