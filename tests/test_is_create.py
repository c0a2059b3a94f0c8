"""Creation of a single-tree importance-sampling handle that is refused."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200.graph import OR, probability_threshold


@pytest.mark.gpu
def test_the_event_limit_is_checked_before_the_buffers(capi, gpu):
    """15,000 events are past the entry point's limit; the chunk asked for would
    take two buffers of 126 GB, which no device has room for, so a check behind
    their allocation answers with the wrong error."""
    from mcscram_b200.importance import BatchedImportanceSampler, ImportanceSampler
    n = 15000
    g = G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n), be_event_idx=np.arange(n),
                    be_threshold=probability_threshold(np.full(n, 1e-4)), gate_op=[OR], gate_k=[0], gate_in_begin=[0],
                    gate_in_count=[n], gate_neg_count=[0], inputs=np.arange(n), tally_nodes=[n])
    with pytest.raises(capi.McgError) as exc:
        ImportanceSampler(g, chunk_words=1 << 20)
    assert exc.value.code == 1 and "too many basic events" in str(exc.value)
    with BatchedImportanceSampler([g], chunk_words=256) as s:  # the entry point for such trees
        assert s.run(g.be_threshold, word_count=4)["hits"][0] > 0
