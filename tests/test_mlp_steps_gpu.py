"""Training steps that overlap on the GPU, with Adam inside the batch sums and
the rounded weights kept up beside them, against the same steps made one by one:
the gradient at the weights so far, and Adam on the host in FP32 with the
kernel's order of operations.  Bit for bit: both sum in the same order, and a
step that read weights, moments or rounded weights of another step would not
give the same bits.  (The products of a fused multiply-add are exact in the
host's long double.)"""
import ctypes
import ctypes.util

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _fma(a, b, c):
    return (np.asarray(a, np.longdouble) * np.asarray(b, np.longdouble) + np.asarray(c, np.longdouble)).astype(F)


def _powf(x, y):
    powf = ctypes.CDLL(ctypes.util.find_library("m") or "libm.so.6").powf
    powf.restype, powf.argtypes = ctypes.c_float, [ctypes.c_float, ctypes.c_float]
    return F(powf(float(x), float(y)))


@pytest.mark.parametrize("batch,batches,epochs", [(257, 5, 2), (1000, 5, 2), (16, 7, 1), (1, 9, 1)])
def test_overlapped_steps_are_the_single_steps(ctx, batch, batches, epochs):
    import vnm_gb300
    rng = np.random.default_rng(batch)
    n = batch * batches
    X = rng.random((n, 32), dtype=np.float32)
    t = (X @ rng.standard_normal(32).astype(F) + 0.3 * rng.standard_normal(n)).astype(F)
    net, one = vnm_gb300.Mlp(ctx, 3), vnm_gb300.Mlp(ctx, 4)
    p = net.get()
    lr, b1, b2, eps = F(2e-3), F(0.9), F(0.999), F(1e-8)
    m, v = np.zeros_like(p), np.zeros_like(p)
    step = 0
    for _ in range(epochs):
        for k in range(batches):
            rows = slice(k * batch, (k + 1) * batch)
            one.set(p)
            g = one.grad(X[rows], t[rows])[0]
            step += 1
            c1, c2 = F(1) - _powf(b1, step), F(1) - _powf(b2, step)
            m = _fma(F(1) - b1, g, b1 * m)
            v = _fma((F(1) - b2) * g, g, b2 * v)
            p = p - lr * (m / c1) / (np.sqrt(v / c2) + eps)
            assert p.dtype == F
    net.train(X, t, batch=batch, epochs=epochs, lr=float(lr))
    assert np.array_equal(net.get().view(np.int32), p.view(np.int32))
