"""The Gauss-Seidel sweep by blocks of rows against the oracle's sequential
sweep, level by level: hierarchies whose levels run in one block and in many,
with one to 32 lanes a row, rows that take several records (over 100 entries),
diagonal-only rows, chunks and BlockSOR blocks.  Integer sweeps and FP sweeps
in the sequential-order mode must match bit for bit.  FP sweeps otherwise differ
in the order of a row's sum: at most (entries + 2) roundings of dinv * (|in| +
sum |l x|), which is at most three times the larger of max|dinv| max|in| and
max|x|; the errors of the rows that a row reads come in scaled by q, its lower
part over its diagonal, so a chain adds up to a factor 1 / (1 - q).  Levels with
q above 0.9 are compared in the sequential-order mode alone."""
import ctypes as C

import numpy as np
import pytest

import oracle_ffi as of
import sagb
import setup_views as sv

pytestmark = pytest.mark.gpu

CASES = [
    (sagb.GEN_POISSON2D, 67, 0.0, {}),
    (sagb.GEN_POISSON2D, 181, 0.0, {}),
    (sagb.GEN_POISSON3D, 33, 0.0, {}),
    (sagb.GEN_POISSON3D, 64, 0.0, {}),
    (sagb.GEN_CONVDIFF3D, 41, 50.0, {}),
    (sagb.GEN_STENCIL27, 40, 0.0, {}),
    (sagb.GEN_ANISO2D, 311, 1e-3, {"smoother_blocks": 40}),
    (sagb.GEN_POISSON3D, 45, 0.0, {"multicolor": 2}),
    (sagb.GEN_POISSON3D, 31, 0.0, {"multicolor": 1}),
]


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


def _setup(kind, n, param, prec, kw):
    A = sagb.HostCsr.generate(kind, n, param, 3)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    r, c, v = A.arrays()
    return sagb.Setup(prec, r, c, v, sagb.amg_params(**kw))


def _levels(ctx, setup, prec, make):
    keep = of.Keep()
    h = sv.oracle_amg(keep, setup)
    cols = sv.colours(setup)
    M = sagb.Amg(ctx, prec, setup=setup)
    suffix = {sagb.INT: "i32", sagb.F64: "f64", sagb.F32: "f32"}[prec]
    ptr = {sagb.INT: of.i32p, sagb.F64: of.f64p, sagb.F32: of.f32p}[prec]
    rng = np.random.default_rng(5)
    for lv in range(setup.depth):
        r = setup.view(sagb.OP_LD, lv)[0]
        x = make(rng, len(r) - 1)
        ref = np.zeros_like(x)
        if cols[lv] is None:
            getattr(of.lib(), f"or_ldtri_{suffix}")(C.byref(h.LD[lv]), None, 0, of.ptr(x, ptr), of.ptr(ref, ptr))
        else:
            order = of.colour_order(cols[lv])
            getattr(of.lib(), f"or_ldtri_order_{suffix}")(C.byref(h.LD[lv]), of.ptr(order, of.i32p), of.ptr(x, ptr),
                                                          of.ptr(ref, ptr))
        for _ in range(2):  # a second sweep meets the first one's published values
            yield lv, x, M.sweep(lv, x), ref
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()


@pytest.mark.parametrize("kind,n,param,kw", CASES)
def test_int_sweeps_bit_exact(ctx, kind, n, param, kw):
    setup = _setup(kind, n, param, sagb.INT, kw)
    for lv, _, got, ref in _levels(ctx, setup, sagb.INT,
                                lambda rng, k: rng.integers(-(1 << 28), 1 << 28, size=k).astype(np.int32)):
        np.testing.assert_array_equal(got, ref, err_msg=f"level {lv}")


@pytest.mark.parametrize("prec,dtype", [(sagb.F64, np.float64), (sagb.F32, np.float32)])
@pytest.mark.parametrize("kind,n,param,kw", CASES[:5] + CASES[6:8])
def test_fp_sweeps(ctx, prec, dtype, kind, n, param, kw):
    setup = _setup(kind, n, param, prec, kw)

    def make(rng, k):
        return rng.standard_normal(k).astype(dtype)

    ctx.set_option(sagb.OPT_FP_EXACT, 1)
    try:
        for lv, _, got, ref in _levels(ctx, setup, prec, make):
            np.testing.assert_array_equal(got, ref, err_msg=f"level {lv}")
    finally:
        ctx.set_option(sagb.OPT_FP_EXACT, 0)
    eps = np.finfo(dtype).eps
    for lv, x, got, ref in _levels(ctx, setup, prec, make):
        r, _, v = setup.view(sagb.OP_LD, lv)[:3]
        lower = np.add.reduceat(np.abs(v.astype(np.float64)), r[:-1]) - np.abs(v[r[1:] - 1])
        q = (lower * np.abs(v[r[1:] - 1])).max()
        if q > 0.9:
            continue
        size = max(np.abs(v[r[1:] - 1]).max() * np.abs(x).max(), np.abs(ref).max())
        tol = 3 / (1 - q) * (np.diff(r).max() + 2) * eps * size
        assert np.abs(got.astype(np.float64) - ref).max() <= tol, f"level {lv}"
