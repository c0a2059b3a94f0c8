"""The proposal network's kernels at the edges of their tiles: rows around a
128-row tile, one and several tiles per CTA, with and without row weights and
on both sides of the row count from which the weights are summed on the
device; and a training step against Adam in numpy on the kernels' gradients."""
import numpy as np
import pytest

from oracle import mlp_oracle


def _rows(n, seed, weights=True):
    rng = np.random.default_rng(seed)
    return (rng.normal(0, 1, (n, 16)).astype(np.float32), rng.uniform(0, 0.5, n).astype(np.float32),
            rng.uniform(0.1, 3, n).astype(np.float32) if weights else None)


def _params(seed):
    rng = np.random.default_rng(seed)
    p = rng.normal(0, 0.2, 16 * 64 + 64 + 64 * 64 + 64 + 64 + 1).astype(np.float32)
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("n,weights", [(1, True), (127, True), (128, False), (129, True), (32767, True), (32768, True),
                                       (37889, False), (75777, True)])
def test_forward_and_gradient_at_tile_edges(gpu, n, weights):
    from mcscram_b200.importance import ProposalMLP
    X, t, w = _rows(n, n, weights)
    params = _params(3)
    m = ProposalMLP()
    m.set_params(params)
    q = m.forward(X)
    g, loss = m.grad(X, t, w)
    g2, loss2 = m.grad(X, t, w)
    m.close()
    # the oracle rounds to BF16 where the kernels do: what is left is FP32 summation and the fast exponential,
    # the bounds of the repository's own test of these kernels
    q_ref, _ = mlp_oracle.forward(params, X, bf=True)
    np.testing.assert_allclose(q, q_ref, atol=2e-3)
    loss_ref, g_ref = mlp_oracle.loss_and_grad(params, X, t, np.ones(n) if w is None else w, bf=True)
    assert loss == pytest.approx(loss_ref, rel=1e-3)
    assert np.linalg.norm(g - g_ref) <= 1e-2 * np.linalg.norm(g_ref)
    assert np.array_equal(g, g2) and loss == loss2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 40000])
def test_training_steps_are_adam_on_the_gradients(gpu, n):
    from mcscram_b200.importance import ProposalMLP
    X, t, w = _rows(n, n)
    p = _params(4)
    a, b = ProposalMLP(), ProposalMLP()
    a.set_params(p)
    m, v = np.zeros(p.size), np.zeros(p.size)
    for k in range(1, 4):
        before = a.params()
        b.set_params(before)  # the gradient at exactly these parameters (it is the same bit for bit)
        g, loss = b.grad(X, t, w)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g.astype(np.float64) ** 2
        want = before - 1e-2 * (m / (1 - 0.9**k)) / (np.sqrt(v / (1 - 0.999**k)) + 1e-8)
        got_loss = a.train(X, t, w, steps=1, lr=1e-2)
        # FP32 parameters below 1 (half an ulp is 6e-8) and updates below 3 lr from FP32 moments
        np.testing.assert_allclose(a.params(), want, rtol=0, atol=5e-7)
        assert got_loss == loss
    # the operand copies the next forward reads follow the trained parameters
    b.set_params(a.params())
    assert np.array_equal(a.forward(X), b.forward(X))
    a.close()
    b.close()
