"""FP64 products are as exact as sums by about three quarters as many lanes as a row
has entries (lane l of G adds entries l, l + G, ... by fused multiply-adds, the lanes
by a butterfly), whatever lanes the kernel uses: on the fine operators of grids, where
one running sum a row is up to 1.4 times as far off.  Both are compared with sums in
extended precision; the two errors' ratio is within two per cent over 50,000 rows and
more, where one that is no larger can come out by chance."""
import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu

CASES = [(sagb.GEN_POISSON2D, 400, 0.0), (sagb.GEN_POISSON2D, 300, 0.0), (sagb.GEN_POISSON3D, 60, 0.0), (sagb.GEN_POISSON3D, 46, 0.0),
         (sagb.GEN_CONVDIFF3D, 60, 50.0), (sagb.GEN_VARCOEF3D, 52, 2.0), (sagb.GEN_STENCIL27, 45, 0.0), (sagb.GEN_STENCIL27, 60, 0.0)]


@pytest.mark.parametrize("kind,n,param", CASES)
def test_error(kind, n, param):
    A = sagb.HostCsr.generate(kind, n, param, 3)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    rptr, cind, val = A.arrays()
    rows = len(rptr) - 1
    x = np.random.default_rng(n).uniform(-1, 1, rows)
    ld = np.longdouble
    prod = val.astype(ld) * x[cind].astype(ld)
    true = np.add.reduceat(prod, rptr[:-1])
    G = 1
    while G < 32 and G < 0.75 * len(cind) / rows:
        G *= 2
    lanes = np.zeros((G, rows))
    lens = np.diff(rptr)
    for k in range(int(lens.max())):
        live = np.nonzero(lens > k)[0]
        lanes[k % G, live] = (prod[rptr[live] + k] + lanes[k % G, live].astype(ld)).astype(np.float64)
    while len(lanes) > 1:
        h = len(lanes) // 2
        lanes = lanes[:h] + lanes[h:]
    ctx = sagb.Context(0)
    M = sagb.Matrix(ctx, sagb.MAT_F64, rptr, cind, val)
    err, ref = (np.sqrt(np.sum(((y - true).astype(np.float64)) ** 2)) for y in (M.spmv(x), lanes[0]))
    assert err <= 1.02 * ref
    M.close()
    ctx.close()
