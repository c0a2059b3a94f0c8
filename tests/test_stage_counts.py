"""k-of-n gates that the staged mode counts in bit slices: remainders of the four
inputs taken at a time, counts of up to eight bits, and their rate."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200.graph import ATLEAST, probability_threshold


def _counting(n_be, n_gates, n_in, layers, seed=0, neg=False):
    """Layers of n/2-of-n gates that read the layer below."""
    rng = np.random.default_rng(seed)
    per = n_gates // layers
    inputs, counts = [], []
    for j in range(n_gates):
        level = min(j // per, layers - 1)
        lo, hi = (0, n_be) if level == 0 else (n_be + (level - 1) * per, n_be + level * per)
        n = int(rng.choice(n_in))
        counts.append(n)
        inputs += [int(x) for x in rng.integers(lo, hi, n)]
    counts = np.array(counts)
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + n_be), be_event_idx=np.arange(n_be),
                       be_threshold=probability_threshold(rng.uniform(0.3, 0.7, n_be)), gate_op=[ATLEAST] * n_gates,
                       gate_k=counts // 2, gate_in_begin=np.concatenate([[0], np.cumsum(counts)[:-1]]),
                       gate_in_count=counts, gate_neg_count=counts // 3 if neg else np.zeros(n_gates),
                       inputs=inputs, tally_nodes=np.arange(n_be, n_be + n_gates))


@pytest.mark.gpu
@pytest.mark.parametrize("words", [37, 9600])
@pytest.mark.parametrize("n_in", [[9, 10, 11], [12, 13], [14, 15, 16], [31, 32, 33], [127, 128, 254, 255]])
def test_counts(capi, oracle_mod, gpu, n_in, words):
    g = _counting(25, 24, n_in, 3, seed=n_in[0], neg=True)
    with capi.Engine(g, mode=capi.MODE_STAGED) as e:
        e.run(2, 1, 5, words)
        ones, _ = e.tallies()
    assert np.array_equal(ones, oracle_mod.tallies(g, 2, 1, 5, words))


@pytest.mark.gpu
def test_counting_is_no_slower_than_in_the_strip_mode(capi, gpu):
    """600 gates of 60 inputs on 131,072 words: 8.4 ms staged and 13.5 in strips
    (one input and 32 bits at a time, staged took 28.8)."""
    g = _counting(200, 600, [60], 4).with_tallies([799])
    ms = {}
    for mode in (capi.MODE_STRIP, capi.MODE_STAGED):
        with capi.Engine(g, mode=mode) as e:
            e.run(1, 1, 0, 1 << 17)
            e.synchronize()
            ms[mode] = min(e.time_runs(2 + r, 0, 1 << 17, 1) for r in range(3))
    assert ms[capi.MODE_STAGED] <= ms[capi.MODE_STRIP]
