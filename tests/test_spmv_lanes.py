"""Lanes per row of the plain SpMV: the rule of host/spmv_lanes.hpp, compiled by
itself.  Rows of about one length get what their average asks for; a row far
longer than the others gets lanes as long as they shorten the product.  On the
GPU, products with such rows against NumPy: integers bit for bit, FP in the
sequential-order mode bit for bit, FP otherwise within the roundings of a sum in
another order."""
import os
import subprocess

import numpy as np
import pytest

import sagb

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = """
#include <cstdio>
#include "host/spmv_lanes.hpp"
int main() {
    int n, longest, most;
    long long nnz;
    while (scanf("%d %lld %d %d", &n, &nnz, &longest, &most) == 4) printf("%d\\n", sagb::spmv_lanes(n, nnz, longest, most));
}
"""


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "sc23-ad_gb300", "csrc"), str(d / "driver.cpp"),
                           "-o", str(d / "driver")])

    def ask(*args):
        return int(subprocess.run([str(d / "driver")], input=" ".join(map(str, args)), text=True, capture_output=True, check=True).stdout)

    return ask


@pytest.mark.parametrize("n,avg,longest,most,want", [
    (2048383, 7, 7, 32, 1), (2048383, 7, 40, 32, 1), (250000, 55, 55, 32, 4), (125000, 81, 200, 32, 8), (2500, 258, 400, 32, 32),
    (20000, 2, 5, 32, 2), (1, 5, 5, 32, 4), (0, 0, 0, 32, 1), (250000, 55, 55, 2, 2)])
def test_even_rows(lanes, n, avg, longest, most, want):
    assert lanes(n, n * avg, longest, most) == want


@pytest.mark.parametrize("n,avg,longest,most,least", [
    (200000, 6, 200000, 32, 32), (200000, 6, 20000, 32, 8), (40000, 60, 40000, 32, 32), (1000000, 4, 200000, 32, 16),
    (200000, 6, 200000, 8, 8), (5000, 6, 5000, 8, 8)])
def test_a_long_row(lanes, n, avg, longest, most, least):
    assert least <= lanes(n, n * avg, longest, most) <= most


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype", [("i32", np.int32), (sagb.MAT_F64, np.float64), (sagb.MAT_F32, np.float32)])
@pytest.mark.parametrize("n,avg,longest", [(20001, 5, 20001), (30000, 2, 3001), (4001, 40, 4001)])
def test_products(kind, dtype, n, avg, longest):
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 2 * avg + 1, size=n)
    lens[[n // 3, n - 1]] = longest, longest - 3
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cind = rng.integers(0, n, size=rptr[-1]).astype(np.int32)
    ctx = sagb.Context(0)
    if dtype == np.int32:
        val, x = rng.integers(-(1 << 16), 1 << 16, size=len(cind)).astype(dtype), rng.integers(-(1 << 16), 1 << 16, size=n).astype(dtype)
        A = sagb.Matrix(ctx, kind, rptr, cind, val, bit=20)
        total = np.concatenate([[0], np.cumsum(val.astype(np.int64) * x[cind])])
        want = (total[rptr[1:]] - total[rptr[:-1]]) >> 20
        np.testing.assert_array_equal(A.spmv(x), want.astype(np.int32))
    else:
        val, x = rng.standard_normal(len(cind)).astype(dtype), rng.standard_normal(n).astype(dtype)
        A = sagb.Matrix(ctx, kind, rptr, cind, val.astype(np.float64))
        prod = val * x[cind]
        want, size = np.zeros(n, dtype), np.zeros(n)
        for i in range(n):
            p = prod[rptr[i]:rptr[i + 1]]
            want[i] = np.add.accumulate(p)[-1] if len(p) else 0
            size[i] = np.abs(p.astype(np.float64)).sum()
        tol = 2 * (lens + 1) * np.finfo(dtype).eps * size
        assert np.all(np.abs(A.spmv(x).astype(np.float64) - want) <= tol)
        ctx.set_option(sagb.OPT_FP_EXACT, 1)
        np.testing.assert_array_equal(A.spmv(x), want)
    A.close()
    ctx.close()
