"""A creation that ran out of device memory leaves nothing behind: the next
engine on the thread runs."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import OR, probability_threshold


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["strip", "staged", "fused", "layered"])
def test_next_engine_runs(capi, oracle_mod, gpu, mode):
    n = 15000  # two chunk buffers of 126 GB
    large = G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n), be_event_idx=np.arange(n),
                        be_threshold=probability_threshold(np.full(n, 1e-4)), gate_op=[OR], gate_k=[0],
                        gate_in_begin=[0], gate_in_count=[n], gate_neg_count=[0], inputs=np.arange(n),
                        tally_nodes=[n])
    with pytest.raises(capi.McgError) as exc:
        capi.Engine(large, mode=capi.MODE_STAGED, layered_max_words=1 << 20)
    assert exc.value.code == 3
    g = synth.config1()
    with capi.Engine(g, mode=capi.MODES[mode]) as e:
        e.run(1, 1, 0, 100)
        ones, _ = e.tallies()
    assert np.array_equal(ones, oracle_mod.tallies(g, 1, 1, 0, 100))
