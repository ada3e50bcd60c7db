"""Contexts that sweep the same small levels at the same time, from a thread each:
sweeps over vectors of at most 150 KiB publish their values through scratch of
their own context, by blocks of rows and level by level alike.  Every result must
be the one of a sweep alone, with and without allocation."""
import threading

import numpy as np
import pytest

import sagb

pytestmark = pytest.mark.gpu

CASES = [(sagb.INT, np.int32, sagb.GEN_POISSON2D, 181, {}), (sagb.F64, np.float64, sagb.GEN_POISSON2D, 130, {}),
         (sagb.F32, np.float32, sagb.GEN_POISSON3D, 30, {}), (sagb.INT, np.int32, sagb.GEN_POISSON2D, 181, {"multicolor": 1}),
         (sagb.F64, np.float64, sagb.GEN_POISSON2D, 130, {"multicolor": 2})]


@pytest.mark.parametrize("prec,dtype,kind,n,kw", CASES)
def test_two_contexts(prec, dtype, kind, n, kw):
    ctxs = [sagb.Context(0), sagb.Context(0)]
    A = sagb.HostCsr.generate(kind, n)
    _, b = A.rhs(3)
    A.lmax1_scaling(b)
    M = sagb.Amg(ctxs[0], prec, *A.arrays(), params=sagb.amg_params(**kw))
    jobs = []
    for lv in range(M.depth):
        rows = M.level_info(sagb.OP_LD, lv)[0]
        assert rows * np.dtype(dtype).itemsize <= 150 * 1024
        for t, ctx in enumerate(ctxs):
            rng = np.random.default_rng(10 * lv + t)
            x = rng.integers(-(1 << 28), 1 << 28, size=rows).astype(dtype) if prec == sagb.INT else rng.standard_normal(rows).astype(dtype)
            jobs.append((t, lv, M.sweep(lv, x), sagb.DeviceArray.from_host(ctx, x), sagb.DeviceArray(ctx, rows, dtype)))
    lib, failed, gate = sagb.lib(), [], threading.Barrier(2)

    def work(t):
        gate.wait()
        for k in range(60):
            for who, lv, want, x, out in jobs:
                if who != t:
                    continue
                call = lib.sa_amg_sweep if k % 2 else lib.sa_amg_sweep_noalloc
                sagb.check(call(ctxs[t].h, M.h, lv, x.ptr, out.ptr))
                if k % 10 == 9:
                    ctxs[t].sync()
                    if not np.array_equal(out.download(), want):
                        failed.append((t, lv, k))

    threads = [threading.Thread(target=work, args=(t,)) for t in (0, 1)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed
    assert all(c.flags() & sagb.FLAG_TIMEOUT == 0 for c in ctxs)
    for job in jobs:
        job[3].close()
        job[4].close()
    M.close()
    for c in ctxs:
        c.close()
