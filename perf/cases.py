"""The work this framework is timed on: what a program that solves sparse
systems with it calls, through the public Python bindings (the C ABI).

Forms ("form" of a case):
  spmv         one matrix-vector product (Matrix.spmv)
  vcycle       one V-cycle of a single system (Amg.precondition)
  solve        one whole FGMRES(m) solve of a single system (Solver.solve)
  batch_vcycle one V-cycle of a batch of systems (Batch / BatchFp.precondition)
  batch_solve  one whole solve of a batch of systems (Batch / BatchFp.solve)
  train        some epochs of the bit selector's network (Mlp.train)

The systems are the synthetic families of the benchmark: Poisson in 2D and 3D,
2D anisotropic diffusion, 3D diffusion with lognormal coefficients, upwinded
convection-diffusion and random 27-point stencils, rows scaled by their
maxima, b = A x* with x* ~ U[-1, 1].
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sc23-ad_gb300"))
import sagb  # noqa: E402

PRECISION = {"int": sagb.INT, "f64": sagb.F64, "f32": sagb.F32}
VALUE = {"int": torch.int32, "f64": torch.float64, "f32": torch.float32}
STORAGE = {"fixed": sagb.MAT_FIXED, "flex": sagb.MAT_FLEX, "f64": sagb.MAT_F64, "f32": sagb.MAT_F32}
STORED = {"fixed": "int", "flex": "int", "f64": "f64", "f32": "f32"}
FRAC_BITS = 29  # what the bit rule gives these systems
# of each family: grid dimensions, entries a row, entries of all coarse
# operators and of all interpolations for each entry of the fine operator
FAMILY = {"poisson2d": (2, 5, 3.2, 0.98), "poisson3d": (3, 7, 4.1, 0.83), "aniso2d": (2, 5, 1.8, 0.6),
          "varcoef3d": (3, 7, 2.0, 0.41), "convdiff3d": (3, 7, 5.1, 0.63), "stencil27": (3, 27, 0.35, 0.145)}


def listed():
    return [
        # the smallest call: the Krylov operator of a 2D system of an odd side, a few microseconds
        {"name": "spmv-fixed-2d-511", "form": "spmv", "family": "poisson2d", "n": 511, "storage": "fixed"},
        # the refinement operator of the largest single system, an odd side
        {"name": "spmv-f64-3d-127", "form": "spmv", "family": "poisson3d", "n": 127, "storage": "f64"},
        # the drop-in preconditioner on a small ragged system: the reference's natural SOR order
        {"name": "vcycle-int-2d-181", "form": "vcycle", "family": "poisson2d", "n": 181, "precision": "int", "smoother": "sor"},
        # the drop-in preconditioner at its headline size
        {"name": "vcycle-int-3d-128", "form": "vcycle", "family": "poisson3d", "n": 128, "precision": "int", "smoother": "sor"},
        # the FP32-mixed sibling with the reference's parallel smoother (BlockSOR-40)
        {"name": "vcycle-f32-block-aniso-383", "form": "vcycle", "family": "aniso2d", "n": 383, "precision": "f32", "smoother": "block40"},
        # whole solves behind the reference's driver, which hands over host vectors: FP64 and integer
        {"name": "solve-f64-convdiff-41", "form": "solve", "family": "convdiff3d", "n": 41, "precision": "f64", "smoother": "sor", "m": 30},
        {"name": "solve-int-varcoef-40", "form": "solve", "family": "varcoef3d", "n": 40, "precision": "int", "smoother": "sor", "m": 30},
        # the batched engine's V-cycle on the headline system, with the colour caps its tuner keeps there
        {"name": "batch-vcycle-int-3d-128", "form": "batch_vcycle", "family": "poisson3d", "lo": 128, "hi": 128, "systems": 1,
         "rhs": 1, "precision": "int", "coarse_colours": 1},
        # many systems of uneven size, four right-hand sides each, the default colour caps
        {"name": "batch-vcycle-int-27pt-24x4", "form": "batch_vcycle", "family": "stencil27", "lo": 16, "hi": 44, "systems": 24,
         "rhs": 4, "precision": "int", "coarse_colours": 2},
        # the headline solve: early restart, explicit residual, one system
        {"name": "batch-solve-int-3d-96", "form": "batch_solve", "family": "poisson3d", "lo": 96, "hi": 96, "systems": 1, "rhs": 1,
         "precision": "int", "coarse_colours": 1, "m": 30},
        # the FP64 sibling on the batched design, nonsymmetric systems, two right-hand sides
        {"name": "batch-solve-f64-convdiff-2x2", "form": "batch_solve", "family": "convdiff3d", "lo": 37, "hi": 57, "systems": 2,
         "rhs": 2, "precision": "f64", "coarse_colours": 2, "m": 30},
        # retraining the bit selector on as many matrices as the committed dataset holds
        {"name": "train-selector-1109", "form": "train", "rows": 1109, "batch": 64, "epochs": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["spmv", "vcycle", "vcycle", "solve", "batch_vcycle", "batch_vcycle", "batch_solve", "batch_solve", "train"])
    if form == "spmv":
        family = rng.choice(["poisson2d", "poisson3d", "varcoef3d", "convdiff3d", "stencil27"])
        rows = _log(rng, 4000, 800000 if family == "stencil27" else 2000000)
        return {"form": form, "family": family, "n": int(rows ** (1.0 / FAMILY[family][0])), "storage": rng.choice(sorted(STORAGE))}
    if form == "train":
        return {"form": form, "rows": _log(rng, 100, 2000), "batch": rng.choice([32, 64, 100]), "epochs": rng.randint(1, 3)}
    precision = rng.choice(["int", "int", "f64", "f32"])
    if form == "vcycle":
        family = rng.choice(sorted(FAMILY))
        rows = _log(rng, 4500, 260000)
        return {"form": form, "family": family, "n": int(rows ** (1.0 / FAMILY[family][0])), "precision": precision,
                "smoother": rng.choice(["sor", "sor", "block40", "chunks", "colours"])}
    # anisotropic systems overflow the integer solver at these bits and go through its fallback
    family = rng.choice(["poisson2d", "poisson3d", "varcoef3d", "convdiff3d", "stencil27"])
    root = 1.0 / FAMILY[family][0]
    if form == "solve":
        rows = _log(rng, 4500, 64000)
        return {"form": form, "family": family, "n": int(rows ** root), "precision": precision,
                "smoother": rng.choice(["sor", "sor", "block40", "chunks"]), "m": rng.choice([20, 30])}
    systems = _log(rng, 1, 32)
    most = min(262144.0, 800000.0 / systems)
    hi = _log(rng, 4500, most)
    lo = _log(rng, 4200, hi)
    case = {"form": form, "family": family, "lo": int(lo ** root), "hi": int(hi ** root), "systems": systems,
            "rhs": rng.choice([1, 1, 2, 4]), "precision": precision, "coarse_colours": rng.choice([1, 2, 2])}
    if form == "batch_solve":
        case["m"] = rng.choice([20, 30])
    return case


# ------------------------------------------------------------------- systems

def _system(family, n, rng):
    """CSR arrays of one system, rows scaled by their maxima."""
    dims = FAMILY[family][0]
    N = n ** dims
    idx = np.arange(N, dtype=np.int32)
    x, y = idx % n, idx // n % n
    z = idx // (n * n) if dims == 3 else None
    cols, vals, keep = [], [], []

    def put(ok, col, val):
        cols.append(np.where(ok, col, 0).astype(np.int32))
        vals.append(np.broadcast_to(np.asarray(val, np.float64), (N,)))
        keep.append(ok)

    everywhere = np.ones(N, bool)
    if family == "stencil27":
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if dx == dy == dz == 0:
                        put(everywhere, idx, 26.0 + rng.uniform(0.1, 1.0, N))
                    else:
                        ok = (x + dx >= 0) & (x + dx < n) & (y + dy >= 0) & (y + dy < n) & (z + dz >= 0) & (z + dz < n)
                        put(ok, idx + dx + n * dy + n * n * dz, -1.0)
    else:
        axes = [(x, 1), (y, n)] + ([(z, n * n)] if dims == 3 else [])
        k = np.exp(2.0 * rng.standard_normal(N)) if family == "varcoef3d" else None
        low, high, diag = [], [], np.zeros(N)
        for a, (pos, step) in enumerate(axes):
            inner, outer = pos > 0, pos < n - 1
            if family == "varcoef3d":  # harmonic means on the faces, the cell's own value on the boundary
                dn, up = np.roll(k, step), np.roll(k, -step)
                wl = np.where(inner, 2.0 * k * dn / (k + dn), k)
                wh = np.where(outer, 2.0 * k * up / (k + up), k)
            elif family == "aniso2d":
                wl = wh = 1.0 if a == 0 else 1e-3
            elif family == "convdiff3d":  # upwinded, Peclet number 50 along the first axis
                wl, wh = (1.0 + 50.0 / n, 1.0) if a == 0 else (1.0, 1.0)
            else:
                wl = wh = 1.0
            diag += wl
            diag += wh
            low.append((inner, idx - step, -np.asarray(wl)))
            high.append((outer, idx + step, -np.asarray(wh)))
        for e in reversed(low):
            put(*e)
        put(everywhere, idx, diag)
        for e in high:
            put(*e)
    keep = np.stack(keep, 1)
    cols, vals = np.stack(cols, 1)[keep], np.stack(vals, 1)
    vals = (vals / np.where(keep, np.abs(vals), 0.0).max(1)[:, None])[keep]
    rptr = np.zeros(N + 1, np.int32)
    np.cumsum(keep.sum(1), out=rptr[1:])
    return rptr, cols, np.ascontiguousarray(vals)


def _times(system, x):
    """A x in 64 bits."""
    r, c, v = system
    return np.add.reduceat(v * x[c], r[:-1])


def _sides(case):
    """The sides of a batch's systems, spread evenly over the case's range."""
    k = case["systems"]
    return [case["lo"] + (case["hi"] - case["lo"]) * i // max(1, k - 1) for i in range(k)]


def _problem(case, seed):
    """The systems of a case and the solutions that its right-hand sides are made from (rows x right-hand sides)."""
    rng = np.random.default_rng(seed)
    sides = _sides(case) if "systems" in case else [case["n"]]
    systems = [_system(case["family"], n, rng) for n in sides]
    sols = [rng.uniform(-1.0, 1.0, (len(s[0]) - 1, case.get("rhs", 1))) for s in systems]
    return systems, sols


def _krylov_vector(rows, rhs, precision, seed):
    """A normalised Krylov vector as FGMRES hands it to the preconditioner or the operator."""
    v = torch.rand(rows, rhs, dtype=torch.float64, generator=torch.Generator().manual_seed(seed)) * 2 - 1
    v /= v.norm(dim=0)
    if precision == "int":
        v = torch.trunc(v * 2.0 ** FRAC_BITS)
    return v.to(VALUE[precision]).reshape(-1).contiguous()


# ------------------------------------------------------------------ the cases

_context = None


def _ctx():
    global _context
    if _context is None:
        torch.cuda.init()
        _context = sagb.Context(0)
    return _context


def _at(t):
    return ctypes.c_void_p(t.data_ptr())


class State:
    """What a program keeps between calls."""

    def __init__(self, case):
        self.case = dict(case)
        self.handles = []  # closed last to first

    def keep(self, handle):
        self.handles.append(handle)
        return handle

    def __del__(self):
        while self.handles:
            self.handles.pop().close()


def _single(s, case, systems):
    smoother = case["smoother"]
    params = sagb.amg_params(smoother_blocks=40 if smoother == "block40" else 0,
                             multicolor={"chunks": 2, "colours": 1}.get(smoother, 0))
    p = PRECISION[case["precision"]]
    setup = sagb.Setup(p, *systems[0], params=params, ctx=_ctx())
    s.amg = s.keep(sagb.Amg(_ctx(), p, setup=setup))
    setup.close()


def _batch(s, case, systems):
    params = sagb.amg_params(max_colours=8, coarse_size=400, coarse_colours=case["coarse_colours"])
    s.engine = s.batch = s.keep(sagb.Batch(_ctx(), systems, case["rhs"], params))
    if case["precision"] != "int":
        s.engine = s.keep(sagb.BatchFp(_ctx(), s.batch, PRECISION[case["precision"]]))
    s.engine.autotune()


def prepare(case, seed):
    s, ctx, form = State(case), _ctx(), case["form"]
    if form == "train":
        rng = np.random.default_rng(seed)
        s.X = rng.standard_normal((case["rows"], 20)).astype(np.float32)
        s.T = rng.uniform(2.0, 11.0, (case["rows"], 22)).astype(np.float32)
        s.M = np.ones_like(s.T)
        s.net = s.keep(sagb.Mlp(ctx, 20, 64, 22, seed=seed))
        s.params = s.net.params()
        return s
    systems, sols = _problem(case, seed)
    if form == "spmv":
        s.matrix = s.keep(sagb.Matrix(ctx, STORAGE[case["storage"]], *systems[0], bit=30))
        s.x = _krylov_vector(s.matrix.m, 1, STORED[case["storage"]], seed).cuda()
        s.y = torch.empty_like(s.x)
    elif form in ("vcycle", "batch_vcycle"):
        (_single if form == "vcycle" else _batch)(s, case, systems)
        rows = sum(len(a[0]) - 1 for a in systems)
        s.x = _krylov_vector(rows, case.get("rhs", 1), case["precision"], seed).cuda()
        s.y = torch.empty_like(s.x)
    else:
        b = [np.stack([_times(a, x[:, k]) for k in range(x.shape[1])], 1) for a, x in zip(systems, sols)]
        s.norms = np.concatenate([np.linalg.norm(v, axis=0) for v in b])
        b = np.concatenate([v.reshape(-1) for v in b])
        if form == "solve":
            _single(s, case, systems)
            p = PRECISION[case["precision"]]
            s.dA = s.keep(sagb.Matrix(ctx, sagb.MAT_F64, *systems[0]))
            kind = {"int": sagb.MAT_FIXED, "f64": sagb.MAT_F64, "f32": sagb.MAT_F32}[case["precision"]]
            s.A = s.keep(sagb.Matrix(ctx, kind, *systems[0], bit=30))
            s.solver = s.keep(sagb.Solver(ctx, p, s.dA, s.A, s.amg, sagb.solver_params(m=case["m"], frac_bits=FRAC_BITS)))
            s.b, s.x = b, np.zeros_like(b)
        else:
            _batch(s, case, systems)
            s.solver_params = sagb.solver_params(m=case["m"], explicit_stop=1, cycle_bits=12)
            s.bits = [FRAC_BITS] * case["systems"]
            s.b = torch.from_numpy(b).cuda()
            s.x = torch.empty_like(s.b)
            s.stream = torch.cuda.ExternalStream(ctx.stream())
    torch.cuda.synchronize()
    return s


def run(s):
    form = s.case["form"]
    if form == "spmv":
        s.matrix.spmv(_at(s.x), _at(s.y))
        return s.y
    if form == "vcycle":
        s.amg.precondition(_at(s.x), _at(s.y))
        return s.y
    if form == "batch_vcycle":
        s.engine.precondition(_at(s.x), _at(s.y))
        return s.y
    if form == "train":
        s.net.set_params(s.params)
        loss = s.net.train(s.X, s.T, s.M, epochs=s.case["epochs"], batch=s.case["batch"], lr=2e-3, seed=1)
        return {"loss": loss, "params": s.net.params()}
    if form == "solve":
        s.x[:] = 0.0
        iters, conv = s.solver.solve(s.b, float(s.norms[0]), s.x)
        return {"x": s.x, "iters": iters, "converged": conv}
    with torch.cuda.stream(s.stream):
        s.x.zero_()
    if s.case["precision"] == "int":
        iters, conv, bits = s.engine.solve(s.solver_params, s.bits, _at(s.b), s.norms, _at(s.x))
        return {"x": s.x, "iters": iters, "converged": conv, "bits": bits}
    iters, conv = s.engine.solve(s.solver_params, _at(s.b), s.norms, _at(s.x))
    return {"x": s.x, "iters": iters, "converged": conv}


def work(case):
    form = case["form"]
    if form == "train":
        weights = 20 * 64 + 64 * 64 + 64 * 22 + 150
        steps = case["epochs"] * -(-case["rows"] // case["batch"])
        return {"bytes": 4 * (case["rows"] * (20 + 2 * 22) + 2 * weights), "flops": 6 * weights * case["rows"] * case["epochs"] + 12 * weights * steps}
    dims, per_row, coarse, interp = FAMILY[case["family"]]
    rows = sum(n ** dims for n in _sides(case)) if "systems" in case else case["n"] ** dims
    rhs, nnz = case.get("rhs", 1), rows * per_row
    if form == "spmv":
        size = 8 if case["storage"] == "f64" else 4
        return {"bytes": nnz * (size + 4) + 4 * (rows + 1) + 2 * size * rows, "flops": 2 * nnz}
    size = 8 if case["precision"] == "f64" else 4
    # one V-cycle: every level's operator, its smoother's two triangles, the interpolations and restrictions, read once
    entries = nnz * (2 * (1 + coarse) + 2 * interp)
    bytes_, flops = entries * (4 + size) + 2 * rows * rhs * size, 2 * entries * rhs
    if form in ("solve", "batch_solve"):
        # some ten steps for a residual of 1e-10, each with a V-cycle, a product with A and the orthogonalisation
        steps = 10
        bytes_ = steps * (bytes_ + nnz * (4 + size) + rows * rhs * size * (steps + 3)) + 16 * rows * rhs
        flops = steps * (flops + 2 * nnz * rhs + 4 * rows * rhs * steps)
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------- in 64 bits

def _train_exact(case, s):
    W = [w.astype(np.float64) for w in np.split(s.params.astype(np.float64), np.cumsum([20 * 64, 64, 64 * 64, 64, 64 * 22, 22])[:-1])]
    W[0], W[2], W[4] = W[0].reshape(64, 20), W[2].reshape(64, 64), W[4].reshape(22, 64)
    m1, m2 = [np.zeros_like(w) for w in W], [np.zeros_like(w) for w in W]
    X, T = s.X.astype(np.float64), s.T.astype(np.float64)
    word, state, losses, t = (1 << 64) - 1, 1, [], 0

    def splitmix():
        nonlocal state
        state = (state + 0x9E3779B97F4A7C15) & word
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & word
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & word
        return z ^ (z >> 31)

    for _ in range(case["epochs"]):
        order = list(range(len(X)))
        for i in range(len(X) - 1, 0, -1):
            j = splitmix() % (i + 1)
            order[i], order[j] = order[j], order[i]
        epoch = []
        for at in range(0, len(X), case["batch"]):
            rows = order[at:at + case["batch"]]
            a0 = X[rows]
            a1 = np.maximum(a0 @ W[0].T + W[1], 0.0)
            a2 = np.maximum(a1 @ W[2].T + W[3], 0.0)
            off = a2 @ W[4].T + W[5] - T[rows]
            epoch.append(np.mean(off * off))
            d3 = 2.0 * off / off.size
            d2 = (d3 @ W[4]) * (a2 > 0)
            d1 = (d2 @ W[2]) * (a1 > 0)
            grads = [d1.T @ a0, d1.sum(0), d2.T @ a1, d2.sum(0), d3.T @ a2, d3.sum(0)]
            t += 1
            for w, g, p, q in zip(W, grads, m1, m2):
                p += 0.1 * (g - p)
                q += 0.001 * (g * g - q)
                w -= 2e-3 * (p / (1.0 - 0.9 ** t)) / (np.sqrt(q / (1.0 - 0.999 ** t)) + 1e-8)
        losses.append(np.mean(epoch))
    return {"loss": np.array(losses), "params": np.concatenate([w.reshape(-1) for w in W])}


def exact(case, seed):
    form = case["form"]
    if form == "train":
        return _train_exact(case, prepare(case, seed))
    if form == "spmv":
        if STORED[case["storage"]] == "int":
            return None  # whole numbers
        systems, _ = _problem(case, seed)
        v = _krylov_vector(len(systems[0][0]) - 1, 1, case["storage"], seed).double().numpy()
        A = systems[0]
        if case["storage"] == "f32":  # the operator is kept in FP32
            A = (A[0], A[1], A[2].astype(np.float32).astype(np.float64))
        return _times(A, v)
    if form in ("vcycle", "batch_vcycle"):
        return None  # defined by the framework's own hierarchy
    _, sols = _problem(case, seed)
    x = np.concatenate([v.reshape(-1) for v in sols])
    none = {"x": x, "iters": None, "converged": None}
    return dict(none, bits=None) if form == "batch_solve" and case["precision"] == "int" else none
