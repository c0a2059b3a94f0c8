"""Importance sampling over odd numbers of words: rows are padded to an even
length, so such passes take the same loads as even ones, and the padding counts
for nothing."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, ATLEAST, OR, probability_threshold


def _shared(seed, n_be, n_gates):
    """A rare-event tree with events read by two gates, which the cut-set component draws."""
    return synth.generate(synth.TreeSpec(n_be=n_be, n_gates=n_gates, mix={AND: 0.6, OR: 0.3, ATLEAST: 0.1},
                                         p_range=(1e-3, 0.2), seed=seed, atleast_n=(3, 4), share_be_frac=0.2,
                                         share_scope=1))


@pytest.mark.gpu
@pytest.mark.parametrize("words,cut", [(1, 1), (255, 31), (9473, 0), (12001, 2049), (19001, 9473)])
def test_one_chunk_equals_many(gpu, words, cut):
    """Chunks of 256 words (one per chunk of odd length at most) and one chunk of them all: the same samples."""
    from mcscram_b200.importance import BatchedImportanceSampler
    trees = [_shared(3, 90, 56), _shared(4, 40, 25)]
    got = []
    for chunk in (256, 20480):
        with BatchedImportanceSampler(trees, chunk_words=chunk) as s:
            p = s.union.quantised_probabilities()
            thr = s.proposal_thresholds(np.clip(p ** 0.6, 1e-6, 0.9))
            got.append(s.run(thr, iteration=3, word_count=words, ce=True, words_cutset=cut, q_cutset=thr))
    a, b = got
    assert np.array_equal(a["hits"], b["hits"]) and a["hits"].sum() > 0
    for k in ("sum_w", "sum_w2", "ce_num"):  # FP64 sums of up to 1.2 million terms in another order
        np.testing.assert_allclose(a[k], b[k], rtol=64 * words * 2.0**-53)
    assert np.array_equal(a["max_log_w"], b["max_log_w"])


@pytest.mark.gpu
def test_odd_lengths_are_as_fast_as_even_ones(gpu):
    """4,000 gates on 20,001 words took 1.2 times as long as on 20,002 with rows of odd length."""
    from mcscram_b200.importance import ImportanceSampler
    rng = np.random.default_rng(2)
    n_be, layers, per = 600, 20, 200
    inputs = []
    for level in range(layers):
        lo, hi = (0, n_be) if level == 0 else (n_be + (level - 1) * per, n_be + level * per)
        inputs += [int(x) for x in rng.integers(lo, hi, 3 * per)]
    inputs += list(range(n_be + (layers - 1) * per, n_be + layers * per))
    n = layers * per + 1
    g = G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n_be), be_event_idx=np.arange(n_be),
                    be_threshold=probability_threshold(np.full(n_be, 0.01)), gate_op=[AND] * (n - 1) + [OR],
                    gate_k=np.zeros(n), gate_in_begin=np.arange(n) * 3, gate_in_count=[3] * (n - 1) + [per],
                    gate_neg_count=np.zeros(n), inputs=inputs, tally_nodes=[n_be + n - 1])
    with ImportanceSampler(g) as s:
        ms = [min(s.run(g.be_threshold, iteration=2 + i, word_count=w)["kernel_ms"] for i in range(10))
              for w in (20001, 20002)]
    assert ms[0] <= 1.08 * ms[1]
