"""The batched FP64 coarsest solve on both sides of its dispatch: a cluster for each
right-hand side up to a third as many systems as SMs, one CTA a system beyond, and
systems of one panel.  Each system's V-cycle against the oracle's FP64 V-cycle."""
import pytest

import sagb
from test_gpu_batch_fp import FP64_TOL, _check_vcycle, _systems, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

KINDS = [(sagb.GEN_POISSON2D, 24, 0.0), (sagb.GEN_POISSON3D, 9, 0.0), (sagb.GEN_CONVDIFF3D, 10, 20.0), (sagb.GEN_POISSON2D, 31, 0.0)]
TINY = [(sagb.GEN_POISSON2D, 7, 0.0), (sagb.GEN_POISSON3D, 4, 0.0)]


@pytest.mark.parametrize("kinds,nsys", [(KINDS, 50), (KINDS, 51), (KINDS, 64), (TINY, 3)])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_systems_and_right_hand_sides(ctx, kinds, nsys, nrhs):  # noqa: F811
    systems, _ = _systems([kinds[k % len(kinds)] for k in range(nsys)])
    B = sagb.Batch(ctx, systems, nrhs)
    F = sagb.BatchFp(ctx, B, sagb.F64)
    _check_vcycle(B, F, sagb.F64, nrhs, nsys + nrhs, FP64_TOL)
    assert ctx.flags(clear=True) & sagb.FLAG_TIMEOUT == 0
    F.close()
    B.close()
