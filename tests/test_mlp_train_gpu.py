"""The proposal network's training kernels at the edges of their tiles
(8-row blocks, 256-row chunks of the sums over the batch), against the numpy
gradient and one numpy step of Adam."""
import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _setup(ctx, B):
    import vnm_gb300
    net = vnm_gb300.Mlp(ctx, 5)
    p = net.get()
    rng = np.random.default_rng(B)
    for a, b in ((mo.OFF_B1, mo.OFF_W2), (mo.OFF_B2, mo.OFF_W3), (mo.OFF_B3, mo.NPARAM)):
        p[a:b] = rng.normal(0, 0.1, b - a)
    net.set(p)
    X = rng.normal(0, 1, (B, mo.F)).astype(np.float32)
    t = rng.normal(0, 2, B).astype(np.float32)
    t[-1] = 4.0 * B  # the last row weighs as much as all others: a lost remainder shows
    return net, p, X, t


@pytest.mark.parametrize("B", [1, 7, 8, 9, 255, 257, 768, 1030])
def test_gradient_and_adam_at_odd_batches(ctx, B):
    net, p, X, t = _setup(ctx, B)
    g, loss = net.grad(X, t)
    wl, wg = mo.loss_grad(p, X, t)
    # FP32 sums of at most 1030 terms, and a BF16 rounding of an activation
    # that falls the other way moves its term by at most 2^-8: 2^-7 of each
    # parameter block's largest entry is above both
    assert abs(loss - wl) <= 2.0 ** -7 * abs(wl)
    edges = [0, mo.OFF_B1, mo.OFF_W2, mo.OFF_B2, mo.OFF_W3, mo.OFF_B3, mo.NPARAM]
    for a, b in zip(edges[:-1], edges[1:]):
        assert np.abs(g[a:b] - wg[a:b]).max() <= 2.0 ** -7 * np.abs(wg[a:b]).max(), (a, b)
    # Adam's first step is lr * g / (|g| + 1e-8); the odd row past the batch is not used
    net.set(p)
    net.train(np.concatenate([X, X[:1]]) if B > 1 else X, np.concatenate([t, t[:1]]) if B > 1 else t, batch=B, lr=0.5)
    step = p.astype(np.float64) - net.get()
    big = np.abs(wg) >= 0.05 * np.abs(wg).max()
    assert big.any()
    np.testing.assert_allclose(step[big], 0.5 * np.sign(wg[big]), rtol=1e-5, atol=1e-6)
    assert np.all(np.abs(step) <= 0.5 + 1e-5)
