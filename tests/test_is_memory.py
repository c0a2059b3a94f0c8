"""Importance-sampling handles and device memory: the hit weights behind the
first chunk buffer shrink where there is no room for them, and the buffers of a
large handle are still kept for the next one."""
import numpy as np
import pytest

from mcscram_b200 import synth
from mcscram_b200.graph import AND, OR, probability_threshold

GIB = 1 << 30


def _trees(n, n_be, n_gates):
    return [synth.generate(synth.TreeSpec(n_be=n_be, n_gates=n_gates, mix={AND: 0.5, OR: 0.5}, p_range=(0.05, 0.5),
                                          seed=40 + k)) for k in range(n)]


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
def test_hit_weights_shrink_where_memory_is_taken(capi, gpu):
    """16 trees and chunks of 2^17 words ask for 1 GiB of weights next to two
    buffers; with room for those and a quarter of a GiB the handle is made with
    the least weights, and several launches per chunk give the same sums."""
    import torch
    from mcscram_b200.importance import BatchedImportanceSampler
    trees = _trees(16, 60, 30)
    words = 1 << 17
    capi.trim_memory()
    with BatchedImportanceSampler(trees) as s:
        nodes, thr = s.union.n_nodes, s.union.be_threshold
        want = s.run(thr, iteration=2, word_count=1000, ce=True)
    capi.trim_memory()
    taken = torch.empty(_free() - 2 * nodes * words * 8 - GIB // 4, dtype=torch.uint8, device="cuda")
    try:
        with BatchedImportanceSampler(trees) as s:
            got = s.run(thr, iteration=2, word_count=1000, ce=True)
    finally:
        del taken
        torch.cuda.empty_cache()
    capi.trim_memory()
    assert np.array_equal(got["hits"], want["hits"]) and np.all(want["hits"] > 0)
    # FP64 sums of up to 64,000 terms in another order
    for k in ("sum_w", "sum_w2", "ce_num"):
        np.testing.assert_allclose(got[k], want[k], rtol=64000 * 2.0**-53)
    assert np.array_equal(got["max_log_w"], want["max_log_w"])


@pytest.mark.gpu
def test_two_largest_default_buffers_are_kept(capi, gpu):
    """16,000 nodes: two buffers of 15.6 GiB, 1 GiB of weights behind the first."""
    from mcscram_b200.importance import BatchedImportanceSampler
    trees = _trees(16, 625, 375)
    capi.trim_memory()
    before = _free()
    with BatchedImportanceSampler(trees) as s:
        nodes = s.union.n_nodes
    kept = before - _free()
    capi.trim_memory()
    assert nodes * (1 << 17) * 8 <= 16 * GIB
    assert kept >= 2 * nodes * (1 << 17) * 8
