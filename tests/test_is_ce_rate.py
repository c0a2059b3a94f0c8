"""Cross-entropy sums of few events that fire often: each warp's share of the
words is a chain of loads, which must not outlast the pass itself."""
import numpy as np
import pytest

from mcscram_b200 import synth
from mcscram_b200.graph import AND, OR


@pytest.mark.gpu
def test_few_dense_events(gpu):
    """60 events at 0.3, 4,096 words: the sums add about 20 us to a pass of about
    55 (131 us when a warp read 256 words one after the other)."""
    from mcscram_b200.importance import ImportanceSampler
    g = synth.generate(synth.TreeSpec(n_be=60, n_gates=32, mix={AND: 0.5, OR: 0.5}, p_range=(1e-3, 1e-1), seed=7,
                                      share_be_frac=0.2))
    with ImportanceSampler(g.with_tallies([g.root])) as s:
        thr = s.proposal_thresholds(np.full(g.n_be, 0.3))
        ms = [min(s.run(thr, iteration=2 + i, word_count=4096, ce=ce)["kernel_ms"] for i in range(20))
              for ce in (False, True)]
    assert ms[1] <= 2.0 * ms[0]
