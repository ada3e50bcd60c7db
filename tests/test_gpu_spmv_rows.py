"""The plain SpMV at every number of lanes a row takes, over rows of 0 to twice
the average number of entries (empty rows, remainders of one to three entries a
lane), rectangular: integers bit for bit against numpy's wrapping 64-bit sum, FP
in the sequential-order mode bit for bit against the sum in order, FP otherwise
within the roundings of a sum in another order: 2 (entries + 1) eps sum|a x|."""
import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu

# rows, average length: 1, 2, 4, 8, 16 and 32 lanes
CASES = [(140001, 3), (70001, 26), (20001, 5), (2003, 7), (9001, 20), (1501, 90), (1, 5)]


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


def _matrix(n, avg):
    rng = np.random.default_rng(n)
    m = n // 2 + 3
    lens = rng.integers(0, 2 * avg + 1, size=n)
    lens[-1] = 0 if n > 1 else avg
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return rng, m, rptr, rng.integers(0, m, size=rptr[-1]).astype(np.int32), lens


def _row_sums(rptr, prod, dtype):
    """Sums of each row's products, one after the other in their order."""
    n = len(rptr) - 1
    acc = np.zeros(n, dtype)
    for k in range(int(np.diff(rptr).max())):
        live = rptr[:-1] + k < rptr[1:]
        acc[live] = acc[live] + prod[rptr[:-1][live] + k]
    return acc


@pytest.mark.parametrize("n,avg", CASES)
def test_int(ctx, n, avg):
    rng, m, rptr, cind, _ = _matrix(n, avg)
    val = rng.integers(-(1 << 24), 1 << 24, size=len(cind)).astype(np.int32)
    x = rng.integers(-(1 << 24), 1 << 24, size=m).astype(np.int32)
    A = sagb.Matrix(ctx, "i32", rptr, cind, val, bit=20, m=m)
    want = (_row_sums(rptr, val.astype(np.int64) * x[cind].astype(np.int64), np.int64) >> 20).astype(np.int32)
    np.testing.assert_array_equal(A.spmv(x), want)
    A.close()
    ctx.flags(clear=True)


@pytest.mark.parametrize("kind,dtype", [(sagb.MAT_F64, np.float64), (sagb.MAT_F32, np.float32)])
@pytest.mark.parametrize("n,avg", CASES)
def test_fp(ctx, kind, dtype, n, avg):
    rng, m, rptr, cind, lens = _matrix(n, avg)
    val = rng.standard_normal(len(cind)).astype(dtype)
    x = rng.standard_normal(m).astype(dtype)
    A = sagb.Matrix(ctx, kind, rptr, cind, val.astype(np.float64), m=m)
    want = _row_sums(rptr, val * x[cind], dtype)
    tol = 2 * (lens + 1) * np.finfo(dtype).eps * _row_sums(rptr, np.abs(val.astype(np.float64) * x[cind]), np.float64)
    assert np.all(np.abs(A.spmv(x).astype(np.float64) - want) <= tol)
    ctx.set_option(sagb.OPT_FP_EXACT, 1)
    try:
        np.testing.assert_array_equal(A.spmv(x), want)
    finally:
        ctx.set_option(sagb.OPT_FP_EXACT, 0)
    A.close()
