"""Batched instances on a device whose memory is nearly taken: where the tile
kernel's rows or records do not fit, the interpreter runs the batch."""
import numpy as np
import pytest

from mcscram_b200 import graph as G

EVENTS = 3000


def _tree():
    """Events only, all tallied: their rows stay to the end, so the tile kernel's
    take 3.5 GB on 148 SMs; the interpreter keeps no value of them."""
    rng = np.random.default_rng(1)
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + EVENTS), be_event_idx=np.arange(EVENTS),
                       be_threshold=rng.integers(1, 1 << 32, EVENTS).astype(np.uint64), gate_op=[], gate_k=[],
                       gate_in_begin=[], gate_in_count=[], gate_neg_count=[], inputs=[], tally_nodes=np.arange(EVENTS))


def _leave(mib):
    """Takes all of the device's free memory but `mib` MiB."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(max(free - (mib << 20), 0), dtype=torch.uint8, device="cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("when", ["rows", "records"])
def test_without_room_for_the_tiles(capi, oracle_mod, gpu, when):
    import torch
    from mcscram_b200.uncertainty import Batch
    g = _tree()
    n = 2000  # of two trees in turn, so that every group has one: 480 MB of records
    rng = np.random.default_rng(2)
    thr = [rng.integers(0, 1 << 32, EVENTS).astype(np.uint64) for _ in range(4)]
    inst_thr = [thr[i % 4] for i in range(n)]
    capi.trim_memory()
    taken = _leave(1024) if when == "rows" else None
    try:
        with Batch([g, g]) as b:
            few = b.run([0, 1, 0], thr[:3], iteration=3, words_per_instance=33)
            if when == "records":
                taken = _leave(256)
            got = b.run([i % 2 for i in range(n)], inst_thr, iteration=3, words_per_instance=33)
            again = b.run([0, 1, 0], thr[:3], iteration=3, words_per_instance=33)
    finally:
        del taken
        torch.cuda.empty_cache()
    want = [int(np.sum(oracle_mod.tallies(g.with_thresholds(t), 3, 1, 0, 33))) for t in thr]
    assert [int(x) for x in few] == want[:3]
    assert [int(x) for x in got] == [want[i % 4] for i in range(n)]
    assert [int(x) for x in again] == want[:3]
