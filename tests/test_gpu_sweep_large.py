"""Sweeps of levels too large for one CTA's vector.  FP32 rows of over 38,400-row
levels keep their order of summation, by blocks of rows and level by level: lane g
of G takes entries g, g + G, ..., lane 0 starts from the input, the lanes are added
by a butterfly, G a quarter of the average row; bit for bit against NumPy (a
multiply-add rounds once: exact in float64, rounded to float32).  And an FP64 level
whose plan has more blocks than the GPU has SMs, in the sequential-order mode bit
for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle_ffi as of
import sagb
import setup_views as sv

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def ctx():
    c = sagb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind,n,kw", [(sagb.GEN_POISSON2D, 210, {}), (sagb.GEN_POISSON2D, 210, {"multicolor": 1}),
                                       (sagb.GEN_STENCIL27, 34, {}), (sagb.GEN_STENCIL27, 34, {"multicolor": 2})])
def test_fp32_order(ctx, kind, n, kw):
    A = sagb.HostCsr.generate(kind, n, 0.0, 3)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    setup = sagb.Setup(sagb.F32, *A.arrays(), sagb.amg_params(**kw))
    r, c, v = setup.view(sagb.OP_LD, 0)[:3]
    rows = len(r) - 1
    assert rows > 38400
    G = 1
    while G < 32 and G < (len(c) / rows - 1) / 4:
        G *= 2
    order = np.argsort(setup.view(sagb.OP_COLOR, 0), kind="stable") if kw else np.arange(rows)
    x = np.random.default_rng(n).standard_normal(rows).astype(f32)
    want = np.zeros(rows, f32)
    for i in order:
        lanes = [0.0] * G
        lanes[0] = float(x[i])
        for k, j in enumerate(range(r[i], r[i + 1] - 1)):
            lanes[k % G] = float(f32(lanes[k % G] - float(v[j]) * float(want[c[j]])))
        while len(lanes) > 1:
            h = len(lanes) // 2
            lanes = [float(f32(p + q)) for p, q in zip(lanes[:h], lanes[h:])]
        want[i] = f32(lanes[0]) * v[r[i + 1] - 1]
    M = sagb.Amg(ctx, sagb.F32, setup=setup)
    for _ in range(2):
        np.testing.assert_array_equal(M.sweep(0, x), want)
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()


def test_more_blocks_than_sms(ctx):
    A = sagb.HostCsr.generate(sagb.GEN_POISSON3D, 128)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    setup = sagb.Setup(sagb.F64, *A.arrays(), ctx=ctx)
    keep = of.Keep()
    h = sv.oracle_amg(keep, setup)
    M = sagb.Amg(ctx, sagb.F64, setup=setup)
    x = np.random.default_rng(1).standard_normal(M.level_info(sagb.OP_LD, 0)[0])
    ref = np.zeros_like(x)
    of.lib().or_ldtri_f64(C.byref(h.LD[0]), None, 0, of.ptr(x, of.f64p), of.ptr(ref, of.f64p))
    M.close()
    ctx.set_option(sagb.OPT_FP_EXACT, 1)
    try:
        M = sagb.Amg(ctx, sagb.F64, setup=setup)
        for _ in range(2):
            np.testing.assert_array_equal(M.sweep(0, x), ref)
    finally:
        ctx.set_option(sagb.OPT_FP_EXACT, 0)
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()
