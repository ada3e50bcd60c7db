"""The coarsest LU solve against the oracle's two triangular solves, at sizes
around the 32-row panels: less than one panel, exact panels, remainders, panels
with and without columns that the other warps of the cluster sum, and more
panels than warps.  Integers, and FP in the sequential-order mode, match bit for
bit.  FP otherwise sums a row in another order: substitution with a triangle T
in any order is exact for some T + dT, |dT| <= g |T| with g = (n + 2) eps / (1 -
(n + 2) eps), so each solve's error is at most 2 |T^-1| g |T| |x| against one
that rounds too, and the backward solve carries the forward one's over.  That bound is
wide for the larger sizes in FP32: the error against a solve in extended precision
is also held to eight times the sequential solve's, or eight eps of the result
where that one is exact."""
import ctypes as C

import numpy as np
import pytest

import oracle_ffi as of
import sagb
import setup_views as sv

pytestmark = pytest.mark.gpu

CASES = [(sagb.GEN_POISSON2D, n, 0.0) for n in (2, 5, 8, 9, 11, 14, 16, 20, 45, 64)] + [(sagb.GEN_CONVDIFF3D, 13, 20.0)]
PREC = {sagb.INT: (np.int32, "i32", of.i32p), sagb.F64: (np.float64, "f64", of.f64p), sagb.F32: (np.float32, "f32", of.f32p)}


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


def _setup(kind, n, param, prec):
    A = sagb.HostCsr.generate(kind, n, param, 3)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    r, c, v = A.arrays()
    return sagb.Setup(prec, r, c, v, sagb.amg_params(max_levels=1))


def _oracle(setup, x):
    _, suffix, ptr = PREC[setup.precision]
    keep = of.Keep()
    h = sv.oracle_amg(keep, setup)
    y, out = np.zeros_like(x), np.zeros_like(x)
    getattr(of.lib(), f"or_ltri_{suffix}")(C.byref(h.LUL), of.ptr(x, ptr), of.ptr(y, ptr))
    getattr(of.lib(), f"or_dutri_{suffix}")(C.byref(h.LUU), of.ptr(y, ptr), of.ptr(out, ptr))
    return y, out


@pytest.mark.parametrize("kind,n,param", CASES)
def test_int_bit_exact(ctx, kind, n, param):
    setup = _setup(kind, n, param, sagb.INT)
    M = sagb.Amg(ctx, sagb.INT, setup=setup)
    rng = np.random.default_rng(n)
    rows = len(setup.view(sagb.OP_LUL)[0]) - 1
    for scale in (1 << 20, 1 << 27):
        x = rng.integers(-scale, scale, size=rows).astype(np.int32)
        np.testing.assert_array_equal(M.coarse_solve(x), _oracle(setup, x)[1])
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()


def _dense(setup, op, lower):
    r, c, v = setup.view(op)[:3]
    n = len(r) - 1
    T = np.zeros((n, n))
    T[np.repeat(np.arange(n), np.diff(r)), c] = v
    if lower:
        np.fill_diagonal(T, 1.0)
    else:
        np.fill_diagonal(T, 1.0 / v[r[:-1]].astype(np.float64))
    return T


def _solve_long(L, U, x):
    L, U, y = L.astype(np.longdouble), U.astype(np.longdouble), x.astype(np.longdouble)
    n = len(y)
    for i in range(n):
        y[i] -= L[i, :i] @ y[:i]
    for i in range(n - 1, -1, -1):
        y[i] = (y[i] - U[i, i + 1:] @ y[i + 1:]) / U[i, i]
    return y


@pytest.mark.parametrize("prec", [sagb.F64, sagb.F32])
@pytest.mark.parametrize("kind,n,param", CASES)
def test_fp(ctx, prec, kind, n, param):
    dtype = PREC[prec][0]
    setup = _setup(kind, n, param, prec)
    M = sagb.Amg(ctx, prec, setup=setup)
    rows = len(setup.view(sagb.OP_LUL)[0]) - 1
    x = np.random.default_rng(n).standard_normal(rows).astype(dtype)
    y, ref = _oracle(setup, x)
    got = M.coarse_solve(x)
    bad = x.copy()
    bad[rows - 1] = np.inf  # no infinity or NaN may reach rows that do not depend on it
    got_bad = M.coarse_solve(bad)
    ctx.set_option(sagb.OPT_FP_EXACT, 1)
    try:
        np.testing.assert_array_equal(M.coarse_solve(x), ref)
        np.testing.assert_array_equal(np.isnan(got_bad), np.isnan(M.coarse_solve(bad)))
    finally:
        ctx.set_option(sagb.OPT_FP_EXACT, 0)
    L, U = _dense(setup, sagb.OP_LUL, True), _dense(setup, sagb.OP_LUU, False)
    g = (rows + 2) * np.finfo(dtype).eps
    g /= 1 - g
    err_y = 2 * g * np.abs(np.linalg.inv(L)) @ (np.abs(L) @ np.abs(y))
    tol = np.abs(np.linalg.inv(U)) @ (err_y + 2 * g * np.abs(U) @ np.abs(ref))
    assert np.all(np.abs(got.astype(np.float64) - ref) <= tol)
    true = _solve_long(L, U, x)
    size = np.linalg.norm(true.astype(np.float64))
    err, err_ref = (np.linalg.norm((v - true).astype(np.float64)) / size for v in (got, ref))
    assert err <= 8 * max(err_ref, np.finfo(dtype).eps)
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()
