"""Which kernel a Gauss-Seidel sweep gets: the host's plan (host/sweep_plan.cpp),
compiled by itself, for triangles whose kernels are far apart: natural orders run
by blocks of rows, few levels of many rows in one CTA or spread over the chip.  On
the GPU, sweeps of small levels in few colours or chunks against the oracle's
sequential sweep, bit for bit (FP in the sequential-order mode), with and without
the static scratch."""
import os
import subprocess

import numpy as np
import pytest

import sagb
from test_gpu_sweep_blocks import _levels, _setup

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "sc23-ad_gb300", "csrc", "host")
DRIVER = """
#include <cstdio>
#include "sweep_plan.hpp"
using namespace sagb;
int main(int, char **a) {
    FILE *f = fopen(a[1], "rb");
    int h[6];
    if (fread(h, 4, 6, f) != 6) return 1;
    const int n = h[0], nnz = h[1], es = h[2], hinted = h[3];
    std::vector<int> rptr(n + 1), cind(nnz + 1), hint(n + 1);
    std::vector<char> val((size_t)(nnz + 1) * es, 0);
    if (fread(rptr.data(), 4, n + 1, f) != (size_t)n + 1 || fread(cind.data(), 4, nnz, f) != (size_t)nnz) return 1;
    if (hinted && fread(hint.data(), 4, n, f) != (size_t)n) return 1;
    SweepLimits lim;
    lim.sms = 152;
    lim.smem = 227 * 1024;
    lim.integer = es == 4;
    lim.lanes = h[4];
    lim.lanes_log = h[5];
    const SweepPlan p = build_sweep_plan(rptr.data(), cind.data(), val.data(), es, n, lim, hinted ? hint.data() : nullptr);
    const long long bytes = p.ok() ? p.stream.back() * p.quads * 512ll : 0;
    printf("%s %d %lld\\n", p.ok() ? "blocks" : p.one_cta ? "cta" : "spread", p.ok() ? p.blocks : p.levels->nlev, bytes);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I" + HOST, str(d / "driver.cpp")]
                          + [os.path.join(HOST, f) for f in ("sweep_plan.cpp", "schedule.cpp", "tri_cost.cpp")] + ["-o", str(d / "driver")])

    def ask(rows, es=4, hint=None, order=False):
        """rows: columns left of the diagonal of each row; order: the order of its sum is given"""
        lens = np.array([len(r) + 1 for r in rows], np.int32)
        rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        cind = np.concatenate([np.append(r, i) for i, r in enumerate(rows)] or [[]]).astype(np.int32)
        lanes = 1
        while lanes < 32 and lanes < (rptr[-1] / max(1, len(rows)) - 1) / 4:
            lanes *= 2
        head = [len(rows), len(cind), es, int(hint is not None), lanes, lanes.bit_length() - 1 if order else -1]
        with open(d / "in", "wb") as f:
            for a in (head, rptr, cind) + (() if hint is None else (hint,)):
                f.write(np.asarray(a, np.int32).tobytes())
        out = subprocess.run([str(d / "driver"), str(d / "in")], capture_output=True, text=True, check=True).stdout.split()
        return out[0], int(out[1]), int(out[2])

    return ask


def _grid(n, dims):
    """The lower neighbours of a grid's cells in their natural order."""
    i = np.arange(n ** dims)
    steps = [n ** k for k in range(dims)]
    return [[c - s for s in reversed(steps) if c // s % n > 0] for c in i]


@pytest.mark.parametrize("es", [4, 8])
def test_natural_orders_run_by_blocks(plan, es):
    for n, dims in ((40, 2), (181, 2), (20, 3), (40, 3)):
        assert plan(_grid(n, dims), es)[0] == "blocks"


@pytest.mark.parametrize("es", [4, 8])
@pytest.mark.parametrize("order", [False, True])
def test_two_colours_run_in_one_cta(plan, es, order):
    n = 60
    i = np.arange(n * n)
    colour = (i % n + i // n) % 2
    near = [[c + s for s, ok in ((-n, c >= n), (-1, c % n > 0), (1, c % n < n - 1), (n, c < n * n - n)) if ok] for c in i]
    assert plan([r if k else [] for r, k in zip(near, colour)], es, colour, order)[:2] == ("cta", 2)
    # the same with the rows in the order of their colours: a lower triangle, no hint
    at = np.argsort(np.argsort(colour, kind="stable"))
    rows = [None] * (n * n)
    for c in i:
        rows[at[c]] = sorted(at[near[c]]) if colour[c] else []
    assert plan(rows, es, None, order)[:2] == ("cta", 2)


def test_chunks_of_a_large_level_are_spread(plan):
    n, chunk = 40, 1200
    rows = [[c for c in r if c // chunk < i // chunk] for i, r in enumerate(_grid(n, 3))]
    assert plan(rows, 4, np.arange(n ** 3) // chunk)[0] == "spread"


def test_edges(plan):
    assert plan([])[0] == "cta"
    assert plan([[]])[1] == 1
    assert plan([[1], []])[0] != "blocks"  # not a lower triangle, no levels given
    assert plan([[1], []], 4, [1, 0])[1] in (1, 2)


SMALL = [(sagb.GEN_POISSON2D, 40, 0.0, {"multicolor": 1}), (sagb.GEN_POISSON2D, 70, 0.0, {"multicolor": 1}),
         (sagb.GEN_POISSON2D, 70, 0.0, {"multicolor": 2}), (sagb.GEN_STENCIL27, 15, 0.0, {"multicolor": 1}),
         (sagb.GEN_POISSON3D, 40, 0.0, {"multicolor": 2}), (sagb.GEN_CONVDIFF3D, 26, 50.0, {"multicolor": 1})]


@pytest.mark.gpu
@pytest.mark.parametrize("prec,dtype", [(sagb.INT, np.int32), (sagb.F64, np.float64), (sagb.F32, np.float32)])
@pytest.mark.parametrize("kind,n,param,kw", SMALL)
def test_sweeps(prec, dtype, kind, n, param, kw):
    ctx = sagb.Context(0)
    setup = _setup(kind, n, param, prec, kw)

    def make(rng, k):
        return rng.integers(-(1 << 28), 1 << 28, size=k).astype(dtype) if prec == sagb.INT else rng.standard_normal(k).astype(dtype)

    ctx.set_option(sagb.OPT_FP_EXACT, 1)
    for lv, x, got, ref in _levels(ctx, setup, prec, make):
        np.testing.assert_array_equal(got, ref, err_msg=f"level {lv}")
    M = sagb.Amg(ctx, prec, setup=setup)
    for lv in range(M.depth):
        x = make(np.random.default_rng(lv), M.level_info(sagb.OP_LD, lv)[0])
        want = M.sweep(lv, x)
        dx, out = sagb.DeviceArray.from_host(ctx, x), sagb.DeviceArray(ctx, len(x), dtype)
        for _ in range(2):
            sagb.check(sagb.lib().sa_amg_sweep_noalloc(ctx.h, M.h, lv, dx.ptr, out.ptr))
            ctx.sync()
            np.testing.assert_array_equal(out.download(), want, err_msg=f"level {lv}")
        dx.close()
        out.close()
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    M.close()
    ctx.close()
