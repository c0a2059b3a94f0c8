"""A network costs little to make: programs make one, train it and drop it."""
import time

import numpy as np
import pytest

from mcscram_b200 import synth


def _least_ms(f, n=30):
    t = []
    for _ in range(n):
        a = time.perf_counter()
        f()
        t.append((time.perf_counter() - a) * 1e3)
    return min(t)


@pytest.mark.gpu
def test_creation_takes_about_as_long_as_a_plain_engine(capi, gpu):
    """Device buffers, a stream and two events either way: 1.5 ms next to 0.9 for
    an engine of the layered mode (2.8 to 4.8 with a page of mapped host memory)."""
    from mcscram_b200.importance import ProposalMLP
    g = synth.config1()
    assert _least_ms(lambda: ProposalMLP().close()) <= 2.5 * _least_ms(
        lambda: capi.Engine(g, mode=capi.MODES["layered"]).close())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 32767, 32768, 32769, 70001])
def test_outputs_on_both_sides_of_the_staged_copy(gpu, n):
    """A short pass reads the flag and the outputs in one copy, a long one in two: the same outputs row by row."""
    from mcscram_b200.importance import ProposalMLP
    x = np.random.default_rng(n).normal(0, 1, (n, 16)).astype(np.float32)
    m = ProposalMLP(seed=5)
    whole = m.forward(x)
    parts = np.concatenate([m.forward(x[i:i + 20000]) for i in range(0, n, 20000)])
    m.close()
    assert whole.shape == (n,) and np.all((whole > 0) & (whole < 1))
    assert np.array_equal(whole, parts)
