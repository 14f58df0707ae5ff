"""Performance cases of the sparse direct solver: numeric factorization and solves of finite-element systems whose
symbolic analysis is kept, as a program that steps, sweeps or iterates over one mesh uses the library.

A case is a dict: "family" (the system), "N" (cells per side; problems for the batch), "do" (what one pass calls),
"precision", "q" (right-hand sides) and, where a program keeps a tuned schedule, "schedule" (the groupBlocks,
smallFront and deferUpdates of analyze). listed() are the measured cases, draw() gives more of the same ranges,
prepare() makes a program's state (plan, factor object, new values and right-hand sides on the GPU), run() is one pass
through the public entry points, work() its unavoidable bytes and flops, exact() the solution in 64 bits by plain
torch (conjugate gradients for the definite systems, a dense factorization for the indefinite ones).
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "applied-multiphysics_b200"))
import ampsolve as amp  # noqa: E402
import batch  # noqa: E402
import workloads as wl  # noqa: E402

GMRES_TOL = 1e-12   # the residual that the benchmark asks of every solution
DENSE_ROWS = 30000  # exact(): the largest indefinite system that is factored densely
LOSS_TANGENT = 0.05  # the lossy Maxwell systems: eps (1 - i tan d)


def listed():
    return [
        # the smallest ordinary use: a 2D study through the class interface with host arrays, latency bound
        {"name": "heat2d-64 class", "family": "heat2d", "N": 64, "do": "class", "precision": "fp64", "q": 1},
        # a time stepper on a 2D mesh: one solve per step with a kept factor (odd size)
        {"name": "heat2d-129 solve", "family": "heat2d", "N": 129, "do": "solve", "precision": "fp64", "q": 1},
        # a small 3D part in FP64, refactored per design step
        {"name": "elastic3d-11 fp64", "family": "elastic3d", "N": 11, "do": "factor_solve", "precision": "fp64", "q": 1},
        # a middle-sized part in mixed precision, default schedule
        {"name": "elastic3d-24 mixed", "family": "elastic3d", "N": 24, "do": "gmres", "precision": "mixed", "q": 1},
        # the benchmark's system, with the schedules that its autotuner settles on
        {"name": "elastic3d-40 fp64", "family": "elastic3d", "N": 40, "do": "factor_solve", "precision": "fp64", "q": 1,
         "schedule": "2,64,2"},
        {"name": "elastic3d-40 mixed", "family": "elastic3d", "N": 40, "do": "gmres", "precision": "mixed", "q": 1,
         "schedule": "2,128,4"},
        # quadratic heat elements, a few load cases, FP64
        {"name": "heat3d-p2-15 fp64", "family": "heat3d_p2", "N": 15, "do": "factor_solve", "precision": "fp64", "q": 5},
        # the largest: quadratic heat elements with the benchmark's 16 load cases, mixed precision and refinement
        {"name": "heat3d-p2-32 mixed", "family": "heat3d_p2", "N": 32, "do": "refined", "precision": "mixed", "q": 16},
        # driven Maxwell with the benchmark's 64 ports: indefinite, LDL^T with a refinement step
        {"name": "maxwell3d-24 ldlt", "family": "maxwell3d", "N": 24, "do": "ldlt", "precision": "fp64", "q": 64},
        # the same physics on a small odd mesh with Bunch-Kaufman pivots and two ports
        {"name": "maxwell3d-13 bk", "family": "maxwell3d", "N": 13, "do": "ldlt-bk", "precision": "fp64", "q": 2},
        # a quarter of the benchmark's batch of independent 2D problems, 1 to 64 right-hand sides each
        {"name": "heat2d-batch-64", "family": "batch", "N": 64, "do": "batch", "precision": "fp64", "q": 64, "sizes": 3},
        # a lossy Maxwell system: complex-symmetric LDL^T through its class with host arrays
        {"name": "maxwell3d-10 complex", "family": "maxwell3d", "N": 10, "do": "complex", "precision": "fp64", "q": 1},
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, int(lo * (hi / lo) ** rng.random() * 1.0001))


def draw(rng: random.Random):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng: random.Random):
    kind = rng.choice(["class", "solve2d", "solve3d", "elastic64", "elasticmx", "heat64", "heatmx", "ldlt", "bk", "batch",
                       "complex"])
    if kind == "class":
        return {"family": "heat2d", "N": _log(rng, 16, 160), "do": "class", "precision": "fp64", "q": 1}
    if kind == "solve2d":
        return {"family": "heat2d", "N": _log(rng, 16, 192), "do": "solve", "precision": "fp64", "q": _log(rng, 1, 64)}
    if kind == "solve3d":
        return {"family": "elastic3d", "N": _log(rng, 6, 28), "do": "solve", "precision": rng.choice(["fp64", "mixed"]),
                "q": _log(rng, 1, 64)}
    if kind == "elastic64":
        return {"family": "elastic3d", "N": _log(rng, 6, 36), "do": "factor_solve", "precision": "fp64",
                "q": _log(rng, 1, 8)}
    if kind == "elasticmx":
        return {"family": "elastic3d", "N": _log(rng, 8, 38), "do": "gmres", "precision": "mixed", "q": 1}
    if kind == "heat64":
        return {"family": "heat3d_p2", "N": _log(rng, 5, 24), "do": "factor_solve", "precision": "fp64",
                "q": _log(rng, 1, 16)}
    if kind == "heatmx":
        return {"family": "heat3d_p2", "N": _log(rng, 6, 28), "do": "refined", "precision": "mixed", "q": _log(rng, 1, 16)}
    if kind == "ldlt":
        return {"family": "maxwell3d", "N": _log(rng, 6, 22), "do": "ldlt", "precision": "fp64", "q": _log(rng, 1, 64)}
    if kind == "bk":
        return {"family": "maxwell3d", "N": _log(rng, 6, 16), "do": "ldlt-bk", "precision": "fp64", "q": _log(rng, 1, 16)}
    if kind == "batch":
        return {"family": "batch", "N": _log(rng, 4, 64), "do": "batch", "precision": "fp64", "q": 64,
                "sizes": rng.randrange(1, 1000)}
    return {"family": "maxwell3d", "N": _log(rng, 5, 12), "do": "complex", "precision": "fp64", "q": 1}


# ---- the systems -----------------------------------------------------------------------------------------------------
def _members(case, seed: int):
    """The batch's problems: sizes from the case, conductivities and right-hand sides from the seed."""
    return [wl.heat2d_lognormal(n, seed + 7919 * i, q)
            for i, (n, q) in enumerate(wl.heat2d_batch_sizes(case["N"], case["sizes"]))]


def _system(case, seed: int):
    """(pattern, values, right-hand sides (q, n), coordinates (x, y, z) of the unknowns) of one seeded system."""
    rng = random.Random(seed)
    s = rng.randrange(1, 1 << 30)
    n, q, family = case["N"], case["q"], case["family"]
    if family == "heat2d":  # lognormal conductivity per triangle
        w = wl.heat2d_lognormal(n, s, q)
    elif family == "elastic3d":  # steel-like to rubber-like homogeneous parts, random body loads
        w = wl.elastic3d(n, E=math.exp(rng.gauss(0.0, 1.0)), nu=rng.uniform(0.2, 0.4), seed=s, q=q)
    elif family == "heat3d_p2":  # conductivity 100 in seeded spheres, 1 elsewhere
        w = wl.heat3d_p2(n, seed=s, q=q)
    elif family == "maxwell3d":  # permittivity 12 in seeded boxes, k^2 between eigenvalues: indefinite
        w = wl.maxwell3d(n, k2=wl.MAXWELL_K2_32, seed=s, q=q)
    else:
        ws = _members(case, s)
        pat, offs, _ = batch.block_diagonal([v.pat for v in ws])
        rhs = np.zeros((max(v.rhs.shape[0] for v in ws), pat.n))
        for v, o in zip(ws, offs):
            rhs[:v.rhs.shape[0], o:o + v.n] = v.rhs
        return pat, np.concatenate([v.values for v in ws]), rhs, None
    return w.pat, w.values, w.rhs, (w.x, w.y, w.z)


def _lossy(case, seed: int):
    """(pattern, Re A, Im A, Re b, Im b, coordinates) of K - k^2 (1 - i tan d) M: M from two values of k^2."""
    rng = random.Random(seed)
    s = rng.randrange(1, 1 << 30)
    k2 = wl.MAXWELL_K2_32
    w, w0 = (wl.maxwell3d(case["N"], k2=k, seed=s, q=2) for k in (k2, 0.0))
    return w.pat, w.values, LOSS_TANGENT * (w0.values - w.values), w.rhs[0].copy(), w.rhs[1].copy(), (w.x, w.y, w.z)


_plans: dict = {}


def _plan(case, pat=None, coords=None):
    """The analysis that a program keeps for one mesh and schedule; values and right-hand sides are new in each state."""
    key = (case["family"], case["N"], case.get("sizes"), case.get("schedule"))
    if key not in _plans:
        if pat is None:
            pat, _, _, coords = _system(dict(case, q=1), 1)
        opts = {}
        if case.get("schedule"):
            g, f, d = (int(v) for v in case["schedule"].split(","))
            opts = {"groupBlocks": g, "smallFront": f, "deferUpdates": d}
        if case["family"] == "heat2d":
            sym = amp.analyze(pat, ordering="amd", **opts)
        elif case["family"] == "batch":
            ws = _members(case, 1)
            perm = np.concatenate([amp.amdOrder(v.pat) + o for v, o in zip(ws, _row_groups(case))]).astype(np.int32)
            sym = amp.analyze(pat, perm=perm, **opts)
        else:
            sym = amp.analyze(pat, ordering="nd3", x=coords[0], y=coords[1], z=coords[2], **opts)
        _plans.clear()  # one mesh at a time
        _plans[key] = sym
    return _plans[key]


def _row_groups(case):
    """First row of each of the batch's problems, and the end."""
    return np.cumsum([0] + [(n - 1) ** 2 for n, _ in wl.heat2d_batch_sizes(case["N"], case["sizes"])])


# ---- a program's state and one pass ------------------------------------------------------------------------------------
def prepare(case, seed):
    do = case["do"]
    if do == "complex":
        pat, re, im, br, bi, coords = _lossy(case, seed)
        return {"do": do, "pat": pat, "re": re, "im": im, "br": br, "bi": bi,
                "num": amp.ComplexSupernodalLDLT(_plan(case, pat, coords))}
    pat, values, rhs, coords = _system(case, seed)
    sym = _plan(case, pat, coords)
    if do == "class":  # host arrays in, host array out
        return {"do": do, "values": values, "b": rhs[0].copy(), "num": amp.SparseCholesky(pat, sym=sym)}
    kind = {"ldlt": amp.LDLT, "ldlt-bk": amp.LDLT_BK}.get(do, amp.CHOLESKY)
    num = amp.NumericFactor(sym, kind, amp.MIXED if case["precision"] == "mixed" else amp.FP64)
    if do == "batch":
        num.set_row_groups(_row_groups(case))
    v = torch.from_numpy(values).cuda()
    b = torch.from_numpy(np.ascontiguousarray(rhs)).cuda()
    state = {"do": do, "num": num, "values": v, "b": b, "x": torch.empty_like(b), "q": int(b.shape[0])}
    torch.cuda.synchronize()
    if do == "solve":  # the factor is kept, the right-hand sides are new
        num.factor((v.data_ptr(), v.numel()), on_device=True)
    return state


def run(state):
    do, num = state["do"], state["num"]
    if do == "class":
        num.factor(state["values"])
        return num.solve(state["b"])
    if do == "complex":
        num.factor(state["re"], state["im"])
        r = num.solveRefined(state["pat"], state["re"], state["im"], state["br"], state["bi"])
        return {"re": r["re"], "im": r["im"]}
    v, b, x, q = state["values"], state["b"], state["x"], state["q"]
    if do == "solve":
        num.solve_device(b.data_ptr(), x.data_ptr(), q)
        return x
    num.factor((v.data_ptr(), v.numel()), on_device=True)
    if do == "factor_solve":
        num.solve_device(b.data_ptr(), x.data_ptr(), q)
        return x
    if do == "gmres":
        num.solve_gmres_ptr(b.data_ptr(), x.data_ptr(), True, tol=GMRES_TOL)
        return x
    num.solve_refined_device(b.data_ptr(), x.data_ptr(), q, maxSteps=10, tol=GMRES_TOL)
    if do in ("ldlt", "ldlt-bk"):
        return {"x": x, "negative": num.nNeg}
    return x


def work(case):
    sym = _plan(case)
    nnz = int(sym.patternKey.split(":")[1])
    n, q = sym.n, case["q"]
    if case["family"] == "batch":
        sizes = wl.heat2d_batch_sizes(case["N"], case["sizes"])
        cc = sym.colCount.astype(np.float64)
        offs = _row_groups(case)
        each = [(o, e, qi) for o, e, (_, qi) in zip(offs[:-1], offs[1:], sizes)]
        return {"bytes": 8.0 * nnz + 16.0 * float(sum((e - o) * qi for o, e, qi in each)),
                "flops": sym.flops + float(sum(4.0 * cc[o:e].sum() * qi for o, e, qi in each))}
    if case["do"] == "solve":  # the factor is an input
        return {"bytes": (4.0 if case["precision"] == "mixed" else 8.0) * sym.nnzL + 16.0 * n * q,
                "flops": 4.0 * sym.nnzL * q}
    if case["do"] == "complex":
        return {"bytes": 16.0 * nnz + 32.0 * n, "flops": 4.0 * (sym.flops + 4.0 * sym.nnzL)}
    return {"bytes": 8.0 * nnz + 16.0 * n * q, "flops": sym.flops + 4.0 * sym.nnzL * q}


# ---- the solutions in 64 bits, by plain torch --------------------------------------------------------------------------
def _conjugate_gradients(A, diag, B, tol=1e-15, most=20000):
    """X (n, q) with A X = B by Jacobi-preconditioned conjugate gradients, twice (the second time on the residual)."""
    X = torch.zeros_like(B)
    for _ in range(2):
        R = B - A @ X
        D = torch.zeros_like(X)
        Z = R / diag
        Pd, rz = Z.clone(), (R * Z).sum(0)
        stop = tol * torch.linalg.norm(B, dim=0)
        for i in range(most):
            if i % 50 == 0 and bool((torch.linalg.norm(R, dim=0) <= stop).all()):
                break
            AP = A @ Pd
            pap = (Pd * AP).sum(0)
            alpha = torch.where(pap > 0, rz / pap, torch.zeros_like(rz))
            D += alpha * Pd
            R -= alpha * AP
            Z = R / diag
            new = (R * Z).sum(0)
            Pd = Z + torch.where(rz > 0, new / rz, torch.zeros_like(rz)) * Pd
            rz = new
        X += D
    return X


def _dense(pat, values, dtype):
    rows = torch.from_numpy(np.repeat(np.arange(pat.n), np.diff(pat.rowptr))).cuda()
    cols = torch.from_numpy(np.asarray(pat.colidx, np.int64)).cuda()
    A = torch.zeros((pat.n, pat.n), dtype=dtype, device="cuda")
    A[rows, cols] = values.cuda()
    return A


def _solve_dense(A, B):
    lu, piv = torch.linalg.lu_factor(A)
    X = torch.linalg.lu_solve(lu, piv, B)
    for _ in range(2):
        X += torch.linalg.lu_solve(lu, piv, B - A @ X)
    return X


def exact(case, seed):
    do = case["do"]
    if do == "complex":
        pat, re, im, br, bi, _ = _lossy(case, seed)
        if pat.n > DENSE_ROWS // 2:
            return None
        A = _dense(pat, torch.complex(torch.from_numpy(re), torch.from_numpy(im)), torch.complex128)
        X = _solve_dense(A, torch.complex(torch.from_numpy(br), torch.from_numpy(bi)).cuda()[:, None])[:, 0]
        return {"re": X.real.cpu().numpy(), "im": X.imag.cpu().numpy()}
    pat, values, rhs, _ = _system(case, seed)
    B = torch.from_numpy(np.ascontiguousarray(rhs.T)).cuda()
    if do in ("ldlt", "ldlt-bk"):
        if pat.n > DENSE_ROWS:
            return None
        X = _solve_dense(_dense(pat, torch.from_numpy(values), torch.float64), B)
        return {"x": X.T.contiguous(), "negative": None}
    rowptr = torch.from_numpy(np.asarray(pat.rowptr, np.int64)).cuda()
    colidx = torch.from_numpy(np.asarray(pat.colidx, np.int64)).cuda()
    v = torch.from_numpy(values).cuda()
    A = torch.sparse_csr_tensor(rowptr, colidx, v, (pat.n, pat.n))
    rows = torch.repeat_interleave(torch.arange(pat.n, device="cuda"), rowptr[1:] - rowptr[:-1])
    diag = v[rows == colidx][:, None]
    X = _conjugate_gradients(A, diag, B).T.contiguous()
    return X[0].cpu().numpy() if do == "class" else X
