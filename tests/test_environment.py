"""The library picks its kernels from the matrices alone: it reads no environment
variables, and a variable of its own prefix changes no result."""
import os
import re

import numpy as np
import pytest

import sagb

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sc23-ad_gb300", "csrc")


def test_sources_read_no_environment():
    found = []
    for folder, _, files in os.walk(CSRC):
        for name in files:
            with open(os.path.join(folder, name), encoding="utf-8") as f:
                found += [f"{name}:{k}" for k, line in enumerate(f, 1) if re.search(r"\b(secure_)?getenv\b", line)]
    assert not found


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", ["1", "2", "x"])
def test_spmv_ignores_the_environment(monkeypatch, lanes):
    n, avg = 1501, 90  # an FP32 row's sum as by 32 lanes
    rng = np.random.default_rng(7)
    lens = rng.integers(0, 2 * avg + 1, size=n)
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cind = rng.integers(0, n, size=rptr[-1]).astype(np.int32)
    val, x = rng.standard_normal(len(cind)), rng.standard_normal(n).astype(np.float32)
    ctx = sagb.Context(0)
    A = sagb.Matrix(ctx, sagb.MAT_F32, rptr, cind, val)
    want = A.spmv(x)
    monkeypatch.setenv("SAGB_GRP", lanes)
    np.testing.assert_array_equal(A.spmv(x), want)
    A.close()
    ctx.close()
