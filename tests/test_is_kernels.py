"""Importance-sampling weights and cross-entropy sums at the edges of their
kernels' tiles: words around a block's four and a warp's share, event counts
around the 128 rows read at a time, every component count, dense and sparse
events, tops that never fire, and a tree wider than a warp."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, ATLEAST, OR, probability_threshold


TWO32 = float(1 << 32)


def _tree(seed, n_be, n_gates, p_range):
    return synth.generate(synth.TreeSpec(n_be=n_be, n_gates=n_gates, mix={AND: 0.4, OR: 0.4, ATLEAST: 0.2},
                                         p_range=p_range, seed=seed, atleast_n=(3, 4)))


def _wide(n, p):
    """OR over n AND pairs: one gate of n gate inputs (more than a warp reads at once)."""
    begin = np.arange(n + 1) * 2
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + 2 * n), be_event_idx=np.arange(2 * n),
                       be_threshold=probability_threshold(np.full(2 * n, p)), gate_op=[AND] * n + [OR],
                       gate_k=np.zeros(n + 1), gate_in_begin=begin, gate_in_count=[2] * n + [n],
                       gate_neg_count=np.zeros(n + 1), inputs=list(range(2 * n)) + list(range(2 * n, 3 * n)),
                       tally_nodes=[3 * n])


def _reference(oracle_mod, u, bb, roots, comps, it):
    """Per-tree sums and CE numerators of the mixture of comps [(thresholds, words)]."""
    p = u.quantised_probabilities()
    n = sum(w for _, w in comps)
    sums, ce, at = np.zeros((len(roots), 4)), np.zeros(u.n_be), 0
    sums[:, 3] = -np.inf
    for thr, w in comps:
        words = oracle_mod.eval_words(u.with_thresholds(thr), it, at, w)
        at += w
        bits = np.unpackbits(words.view(np.uint8).reshape(u.n_nodes, -1), axis=1, bitorder="little").astype(bool)
        for k, root in enumerate(roots):
            s = slice(int(bb[k]), int(bb[k + 1]))
            hit = np.nonzero(bits[root])[0]
            x = bits[s][:, hit]
            lq = []
            for t, wc in comps:
                q = t[s] / TWO32
                a = np.log(p[s] / q) - (np.log1p(-p[s]) - np.log1p(-q))
                lq.append(np.log(wc / n) - (a @ x + np.sum(np.log1p(-p[s]) - np.log1p(-q))))
            lw = -np.logaddexp.reduce(lq, axis=0)
            wv = np.exp(lw)
            sums[k] += [wv.sum(), (wv * wv).sum(), hit.size, 0]
            sums[k, 3] = max(sums[k, 3], lw.max(initial=-np.inf))
            ce[s] += x @ wv
    return sums, ce


@pytest.mark.gpu
@pytest.mark.parametrize("words,n_def", [((1,), 0), ((3,), 0), ((4,), 0), ((5,), 0), ((257,), 0), ((129, 1), 1),
                                         ((31, 33, 2), 2), ((8, 7, 6, 5, 4), 4), ((40,) * 8, 7), ((5000,), 0)])
def test_weights_at_tile_edges(oracle_mod, gpu, words, n_def):
    from mcscram_b200.importance import BatchedImportanceSampler
    # 127, 128, 129 and 300 events; a dense proposal, and a top event that cannot fire
    trees = [_tree(1, 127, 60, (0.01, 0.6)), _tree(2, 128, 64, (0.3, 0.6)), _tree(3, 129, 60, (0.02, 0.3)),
             _tree(4, 300, 150, (0.01, 0.4)), _wide(40, 1e-9)]
    rng = np.random.default_rng(5)
    with BatchedImportanceSampler(trees, chunk_words=4096) as s:
        u, bb, roots = s.union, s.be_begin, s.roots
        p = u.quantised_probabilities()
        comps = [probability_threshold(np.clip(p * rng.uniform(0.7, 1.4, p.size), 1e-9, 0.95)) for _ in words]
        got = s.run(comps[0], iteration=3, word_count=sum(words), ce=True,
                    **(dict(q_defensive=np.array(comps[1:]), words_defensive=list(words[1:])) if n_def else {}))
        plain = s.run(comps[0], iteration=3, word_count=sum(words),
                      **(dict(q_defensive=np.array(comps[1:]), words_defensive=list(words[1:])) if n_def else {}))
    sums, ce = _reference(oracle_mod, u, bb, roots, list(zip(comps, words)), 3)
    assert np.array_equal(got["hits"], sums[:, 2].astype(np.int64))
    # FP64 sums of at most 320,000 terms whose exponents add 300 logarithms
    np.testing.assert_allclose(got["sum_w"], sums[:, 0], rtol=1e-10)
    np.testing.assert_allclose(got["sum_w2"], sums[:, 1], rtol=1e-10)
    np.testing.assert_allclose(got["ce_num"], ce, rtol=1e-10)
    np.testing.assert_allclose(got["max_log_w"], sums[:, 3], rtol=0, atol=1e-10)
    np.testing.assert_allclose(plain["sum_w"], sums[:, 0], rtol=1e-10)
    assert got["hits"][4] == 0 and got["sum_w"][4] == 0 and np.all(got["ce_num"][bb[4]:] == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("n,words", [(31, 7), (32, 8), (33, 9), (70, 33)])
def test_cut_counts_of_a_gate_wider_than_a_warp(oracle_mod, gpu, n, words):
    """All words from the cut-set component: w = S / N(x) with N the number of
    pairs that fired, known in closed form from the sample's own bits."""
    from mcscram_b200.importance import BatchedImportanceSampler
    with BatchedImportanceSampler([_wide(n, 0.2)], chunk_words=256) as s:
        u = s.union
        r = s.run(u.be_threshold, iteration=2, word_count=words, words_cutset=words)
    p = float(u.quantised_probabilities()[0])
    S, m = n * p * p, words * 64
    # every sample holds the forced pair and Binomial(n - 1, p^2) others:
    # E[1 / N] = (1 - (1 - p^2)^n) / (n p^2), so the mean weight is P(top)
    exact = 1.0 - (1.0 - p * p) ** n
    assert r["hits"][0] == m
    assert r["max_log_w"][0] <= np.log(S) + 1e-12
    se = np.sqrt(max(r["sum_w2"][0] / m - (r["sum_w"][0] / m) ** 2, 0.0) / m)
    assert abs(r["sum_w"][0] / m - exact) <= 5 * se + 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("words", [1, 33, 300])
def test_single_tree_run_equals_the_batch_of_one(gpu, words):
    from mcscram_b200.importance import BatchedImportanceSampler, ImportanceSampler
    g = _tree(9, 200, 90, (0.02, 0.4))
    thr = probability_threshold(np.clip(g.quantised_probabilities() * 1.3, 1e-9, 0.9))
    with ImportanceSampler(g) as a, BatchedImportanceSampler([g]) as b:
        x, y = a.run(thr, iteration=4, word_count=words, ce=True), b.run(thr, iteration=4, word_count=words, ce=True)
    assert x["hits"] == y["hits"][0] > 0
    np.testing.assert_allclose([x["sum_w"], x["sum_w2"], x["max_log_w"]],
                               [y["sum_w"][0], y["sum_w2"][0], y["max_log_w"][0]], rtol=1e-12)
    np.testing.assert_allclose(x["ce_num"], y["ce_num"], rtol=1e-12)
