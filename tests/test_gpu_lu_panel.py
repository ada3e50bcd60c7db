"""FP64 coarsest solves of at most 32 rows take each row's entries in the order of
their columns, one fused multiply-add each, and multiply by the inverse diagonal at
the end: bit for bit against the same in exact arithmetic, rounded step by step.
One row more goes another way and stays within the rounding of a sum."""
from fractions import Fraction as F

import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu


def _dense(setup, op):
    r, c, v = setup.view(op)[:3]
    T = np.zeros((len(r) - 1, len(r) - 1))
    T[np.repeat(np.arange(len(r) - 1), np.diff(r)), c] = v
    return T, v[r[:-1]]


@pytest.mark.parametrize("grid", [2, 5, 6, 7, 8, 9])
def test_one_panel(grid):
    ctx = sagb.Context(0)
    A = sagb.HostCsr.generate(sagb.GEN_POISSON2D, grid)
    _, b = A.rhs(1)
    A.lmax1_scaling(b)
    setup = sagb.Setup(sagb.F64, *A.arrays(), sagb.amg_params(max_levels=1))
    M = sagb.Amg(ctx, sagb.F64, setup=setup)
    (L, _), (U, dinv) = _dense(setup, sagb.OP_LUL), _dense(setup, sagb.OP_LUU)
    n = len(dinv)
    x = np.random.default_rng(grid).standard_normal(n)
    y = [0.0] * n
    for i in range(n):
        t = x[i]
        for c in range(i):
            t = float(F(t) - F(L[i, c]) * F(y[c]))
        y[i] = t
    z = [0.0] * n
    for i in range(n - 1, -1, -1):
        t = y[i]
        for c in range(n - 1, i, -1):
            t = float(F(t) - F(U[i, c]) * F(z[c]))
        z[i] = float(F(t) * F(dinv[i]))
    got, want = M.coarse_solve(x), np.array(z)
    if n <= 32:
        np.testing.assert_array_equal(got, want)
    else:
        assert np.abs(got - want).max() <= 4 * (n + 2) * np.finfo(float).eps * np.abs(np.linalg.inv(np.triu(U, 1) + np.diag(1 / dinv))).sum(1).max() * np.abs(x).sum()
    M.close()
    ctx.close()
