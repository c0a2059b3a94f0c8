"""Importance-sampling handles and device memory: the buffers of a large handle
are kept for the next one, with the hit weights behind the first of them."""
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
