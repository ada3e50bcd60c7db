"""Training rounds the same way in every kernel: the weights after some steps, in one
launch per epoch and by separate kernels, bit for bit against Adam in float32 NumPy
on the gradients that the gradient call gives (it sums in the same order), with the
moments' multiply-adds fused as m1 = fma(1 - b1, g, b1 m1), m2 = fma((1 - b2) g, g,
b2 m2).  (A fused product is exact in float64; its sum is rounded to float32 a second
time, which matters in about one of 2^28.)"""
import ctypes

import numpy as np
import pytest

import mlp_oracle as mo
import sagb

pytestmark = pytest.mark.gpu
f = np.float32


@pytest.mark.parametrize("nin,hid,nout,rows,batch", [(20, 64, 22, 200, 64), (7, 33, 5, 51, 25), (20, 100, 22, 60, 25)])
def test_weights(nin, hid, nout, rows, batch):
    libm = ctypes.CDLL("libm.so.6")
    libm.powf.restype, libm.powf.argtypes = ctypes.c_float, [ctypes.c_float, ctypes.c_float]
    ctx = sagb.Context(0)
    rng = np.random.default_rng(rows)
    X, T = rng.standard_normal((rows, nin)).astype(f), rng.standard_normal((rows, nout)).astype(f)
    M = (rng.random((rows, nout)) > 0.3).astype(f)
    net, other = (sagb.Mlp(ctx, nin, hid, nout, seed=2) for _ in range(2))
    w = net.params()
    net.train(X, T, M, epochs=1, batch=batch, lr=1e-2, seed=5)
    gen = mo.splitmix64_stream(5)
    perm = np.arange(rows)
    for i in range(rows - 1, 0, -1):
        j = next(gen) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    b1, b2, one, lr = f(0.9), f(0.999), f(1), f(1e-2)
    m1, m2 = np.zeros_like(w), np.zeros_like(w)

    def fma(a, b, c):
        return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f)

    for t, off in enumerate(range(0, rows, batch), 1):
        idx = perm[off:off + batch]
        other.set_params(w)
        _, g = other.gradient(X[idx], T[idx], M[idx])
        m1 = fma(one - b1, g, b1 * m1)
        m2 = fma((one - b2) * g, g, b2 * m2)
        c1, c2 = one - f(libm.powf(b1, f(t))), one - f(libm.powf(b2, f(t)))
        w = w - lr * (m1 / c1) / (np.sqrt(m2 / c2) + f(1e-8))
    assert t > 2
    np.testing.assert_array_equal(net.params(), w)
    net.close()
    other.close()
    ctx.close()
