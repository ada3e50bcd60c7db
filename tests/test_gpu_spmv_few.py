"""Rows of about as many entries as lanes, and of few entries by one lane: lane g of G
adds entries g, g + G, ... by fused multiply-adds and the lanes are added by a butterfly,
bit for bit, whatever the kernel does with a lane's last entries.  G = 2 stands for one
lane with two sums in turn.  FP64 multiply-adds are taken in extended precision (wider
than a product where long double is, else a rounding away from it in about one sum of
2^11: those rows are held to one unit in the last place)."""
import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu
ld = np.longdouble


@pytest.mark.parametrize("kind,dtype,n,most,G", [
    (sagb.MAT_F64, np.float64, 150001, 4, 2),  # one lane, pair by pair
    (sagb.MAT_F64, np.float64, 150001, 1, 1),
    (sagb.MAT_F64, np.float64, 12001, 14, 8),
    (sagb.MAT_F64, np.float64, 12001, 18, 8),
    (sagb.MAT_F64, np.float64, 2003, 41, 16),
    (sagb.MAT_F64, np.float64, 2003, 90, 32),  # rows on both sides of two entries a lane
    (sagb.MAT_F32, np.float32, 20001, 440, 32),  # all lanes of the order
])
def test_order(kind, dtype, n, most, G):
    rng = np.random.default_rng(most)
    lens = rng.integers(0, most + 1, size=n)
    lens[:3] = 0, most, 1
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cind = rng.integers(0, n, size=rptr[-1]).astype(np.int32)
    val, x = rng.standard_normal(len(cind)).astype(dtype), rng.standard_normal(n).astype(dtype)
    wide = np.float64 if dtype == np.float32 else ld
    lanes = np.zeros((G, n), dtype)
    for k in range(most):
        rows = np.nonzero(lens > k)[0]
        j = rptr[rows] + k
        lanes[k % G, rows] = (val[j].astype(wide) * x[cind[j]].astype(wide) + lanes[k % G, rows].astype(wide)).astype(dtype)
    while len(lanes) > 1:
        h = len(lanes) // 2
        lanes = lanes[:h] + lanes[h:]
    ctx = sagb.Context(0)
    A = sagb.Matrix(ctx, kind, rptr, cind, val.astype(np.float64))
    got = A.spmv(x)
    if dtype == np.float32 or np.finfo(ld).nmant >= 2 * np.finfo(dtype).nmant + 1:
        np.testing.assert_array_equal(got, lanes[0])
    else:
        assert np.all(np.abs(got - lanes[0]) <= np.finfo(dtype).eps * np.bincount(np.repeat(np.arange(n), lens), np.abs(val * x[cind]), n))
    A.close()
    ctx.close()
