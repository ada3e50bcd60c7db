"""FP32 rows keep one order of summation: lane g of G takes entries g, g + G, ...
and the lanes are added by a butterfly, G from the matrix alone, however many lanes
the kernels use.  SpMV and Gauss-Seidel sweeps are compared bit for bit with that
order in NumPy.  A multiply-add rounds once: the product is exact in float64, and
the float64 sum is rounded to float32 (a second rounding that matters in about one
sum of 2^28)."""
import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f32)


def _butterfly(lanes):  # (G, ...) -> sum as lane 0 has it
    while len(lanes) > 1:
        h = len(lanes) // 2
        lanes = lanes[:h] + lanes[h:]
    return lanes[0]


@pytest.mark.parametrize("n,avg", [(150001, 2), (140001, 3), (70001, 26), (20001, 5), (2003, 7), (9001, 20), (1501, 90)])
def test_spmv(ctx, n, avg):
    rng = np.random.default_rng(avg)
    m = n // 2 + 3
    lens = rng.integers(0, 2 * avg + 1, size=n)
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cind = rng.integers(0, m, size=rptr[-1]).astype(np.int32)
    val, x = rng.standard_normal(len(cind)).astype(f32), rng.standard_normal(m).astype(f32)
    G = 1
    while G < 32 and G < 0.75 * len(cind) / n:
        G *= 2
    acc = np.zeros((G, n), f32)
    for k in range(int(lens.max())):
        rows = np.nonzero(lens > k)[0]
        j = rptr[rows] + k
        acc[k % G, rows] = _fma(val[j], x[cind[j]], acc[k % G, rows])
    A = sagb.Matrix(ctx, sagb.MAT_F32, rptr, cind, val.astype(np.float64), m=m)
    np.testing.assert_array_equal(A.spmv(x), _butterfly(acc))
    A.close()


@pytest.mark.parametrize("kind,n,kw", [(sagb.GEN_POISSON2D, 45, {}), (sagb.GEN_STENCIL27, 13, {}), (sagb.GEN_POISSON3D, 16, {}),
                                       (sagb.GEN_POISSON3D, 14, {"multicolor": 2})])
def test_sweeps(ctx, kind, n, kw):
    A = sagb.HostCsr.generate(kind, n, 0.0, 3)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    setup = sagb.Setup(sagb.F32, *A.arrays(), sagb.amg_params(coarse_size=60, **kw))
    M = sagb.Amg(ctx, sagb.F32, setup=setup)
    rng = np.random.default_rng(n)
    for lv in range(setup.depth):
        r, c, v = setup.view(sagb.OP_LD, lv)[:3]
        rows = len(r) - 1
        order = np.arange(rows)
        if kw:
            order = np.argsort(setup.view(sagb.OP_COLOR, lv), kind="stable")
        G = 1
        while G < 32 and G < (len(c) / rows - 1) / 4:
            G *= 2
        x = rng.standard_normal(rows).astype(f32)
        want = np.zeros(rows, f32)
        for i in order:
            lanes = np.zeros(G, f32)
            lanes[0] = x[i]
            for k, j in enumerate(range(r[i], r[i + 1] - 1)):
                lanes[k % G] = f32(np.float64(lanes[k % G]) - np.float64(v[j]) * np.float64(want[c[j]]))
            want[i] = _butterfly(lanes) * v[r[i + 1] - 1]
        np.testing.assert_array_equal(M.sweep(lv, x), want, err_msg=f"level {lv}")
    M.close()
