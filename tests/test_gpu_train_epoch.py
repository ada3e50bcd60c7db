"""Training in one launch per epoch: its mini-batch steps against the same steps
taken one by one (the gradient call sums in the same order, so gradients are
equal), with Adam in float32 NumPy: rows fewer than CTAs, uneven blocks of rows,
a last batch of one row, layers of odd widths, and a net too wide for the launch.
Each step's Adam expression may round differently by a few units in the last
place: 8 eps of lr and of the parameter a step."""
import numpy as np
import pytest

import mlp_oracle as mo
import sagb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("nin,hid,nout,rows,batch", [
    (20, 64, 22, 64, 64), (20, 64, 22, 3, 8), (20, 64, 22, 65, 64), (7, 33, 5, 100, 100), (7, 33, 5, 51, 25),
    (1, 1, 1, 9, 4), (20, 65, 22, 27, 13), (20, 128, 22, 40, 32)])
def test_steps(ctx, nin, hid, nout, rows, batch):
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, nin)).astype(np.float32)
    T = rng.standard_normal((rows, nout)).astype(np.float32)
    M = (rng.random((rows, nout)) > 0.3).astype(np.float32)
    mu, sd = X.mean(0), X.std(0) + np.float32(0.1)
    lr, seed = np.float32(1e-2), 5
    net, other = (sagb.Mlp(ctx, nin, hid, nout, seed=2) for _ in range(2))
    net.set_norm(mu, sd)
    other.set_norm(mu, sd)
    p0 = net.params()
    hist = net.train(X, T, M, epochs=1, batch=batch, lr=float(lr), seed=seed)
    gen = mo.splitmix64_stream(seed)
    perm = np.arange(rows)
    for i in range(rows - 1, 0, -1):
        j = next(gen) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    got = net.params()
    f = np.float32
    b1, b2, one = f(0.9), f(0.999), f(1)
    w, m1, m2, losses = p0.copy(), np.zeros_like(p0), np.zeros_like(p0), []
    for t, off in enumerate(range(0, rows, batch), 1):
        idx = perm[off:off + batch]
        other.set_params(w)
        loss, g = other.gradient(X[idx], T[idx], M[idx])
        losses.append(loss)
        m1 = b1 * m1 + (one - b1) * g
        m2 = b2 * m2 + (one - b2) * g * g
        w = w - lr * (m1 / (one - b1 ** f(t))) / (np.sqrt(m2 / (one - b2 ** f(t))) + f(1e-8))
    if len(losses) == 1:
        assert hist[0] == pytest.approx(losses[0], rel=1e-6)
        assert np.all(np.abs(got - w) <= 8 * np.finfo(f).eps * (lr + np.abs(w)))
    else:  # rounding differences of a step reach the next steps' gradients
        assert hist[0] == pytest.approx(np.mean(losses), rel=1e-4)
        assert np.abs(got - w).max() <= 2e-4
    net.close()
    other.close()
