"""The performance cases of the solve engine: what its users have it do, through the Python API.

Every case goes through the public classes of hsps_b200 -- SparseMatrix.spmv, the
preconditioners, SolverFactory's solvers, AdaptiveSelector, BatchSolver -- on synthetic
systems: the 5-point operators of hsps_b200.problems (constant and lognormal coefficients,
upwind convection-diffusion, shifted Helmholtz) built here on the GPU, and an unstructured
CSR matrix such as a MatrixMarket file gives.  A program keeps its matrix (SparseMatrix)
between calls and pays for preconditioner setup and solve with each system, so a solve case
times both; vectors are host arrays or CUDA tensors, as its callers have them.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) matrix, vectors and handles a program has in hand
    run(state)          one pass, its outputs
    work(case)          bytes and flops the pass cannot do without
    exact(case, seed)   the outputs in plain 64-bit arithmetic, without the engine
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "hybrid-sparse-pde-solver_b200"))
import hsps_b200 as H  # noqa: E402
from hsps_b200 import batch as B  # noqa: E402

F64 = torch.float64


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one product with a matrix that fits any cache: the call's own latency
        {"name": "spmv poisson 64", "kind": "spmv", "problem": "poisson", "side": 64},
        # the largest grid operator in use, 21 M entries: a product at memory bandwidth
        {"name": "spmv varkappa 2048", "kind": "spmv", "problem": "varkappa", "side": 2048},
        # an unstructured matrix as read from a MatrixMarket file: ragged rows of 1 to ~100
        # entries, columns scattered around the diagonal
        {"name": "spmv ragged 300k", "kind": "spmv", "problem": "ragged", "rows": 300007,
         "mean": 24},
        # the smallest complete solve: host vectors, PCG + Jacobi, the default tolerance
        {"name": "cg jacobi 64", "kind": "solve", "solver": "CG", "precond": "JACOBI",
         "problem": "poisson", "side": 64, "tol": 1e-8, "mixed": False, "host": True},
        # a long Krylov iteration in FP64 on an odd grid, vectors resident on the device
        {"name": "cg jacobi 701", "kind": "solve", "solver": "CG", "precond": "JACOBI",
         "problem": "varkappa", "side": 701, "tol": 1e-10, "mixed": False, "host": False},
        # nonsymmetric: convection-diffusion, FGMRES(30) + ILU(0), host vectors
        {"name": "fgmres ilu0 512", "kind": "solve", "solver": "FGMRES", "precond": "ILU",
         "problem": "convdiff", "peclet": 10.0, "side": 512, "tol": 1e-8, "mixed": False,
         "host": True, "drop_tol": 0.0, "restart": 30},
        # the factory's default ILU (threshold 1e-4) on a smaller nonsymmetric system
        {"name": "fgmres ilut 181", "kind": "solve", "solver": "FGMRES", "precond": "ILU",
         "problem": "convdiff", "peclet": 0.1, "side": 181, "tol": 1e-8, "mixed": False,
         "host": False, "drop_tol": 1e-4, "restart": 50},
        # PCG + smoothed aggregation with the library's defaults, FP64, host vectors
        {"name": "cg amg fp64 240", "kind": "solve", "solver": "CG", "precond": "AMG",
         "problem": "varkappa", "side": 240, "tol": 1e-10, "mixed": False, "host": True},
        # the headline system: 4.2 M unknowns, mixed precision, hierarchy cut where it stalls
        {"name": "cg amg mixed 2048", "kind": "solve", "solver": "CG", "precond": "AMG",
         "problem": "varkappa", "side": 2048, "tol": 1e-10, "mixed": True, "host": False,
         "cut": True},
        # the V-cycle by itself, as the preconditioner of a caller's own Krylov loop
        {"name": "vcycle 1024", "kind": "vcycle", "problem": "varkappa", "side": 1024},
        # many uneven small systems in one call, half symmetric, half not, host arrays
        {"name": "batch 384", "kind": "batch", "systems": 384, "lo": 16, "hi": 128},
        # one request of a service: features, solver choice and solve, mixed precision
        {"name": "ladder convdiff 256", "kind": "ladder", "problem": "convdiff", "peclet": 30.0,
         "side": 256, "tol": 1e-10, "mixed": True, "host": True},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def problem(kinds, c):
        c["problem"] = rng.choice(kinds)
        if c["problem"] == "convdiff":
            c["peclet"] = round(math.exp(rng.uniform(0.0, math.log(100.0))), 3)
        return c

    kind = rng.choice(["spmv", "spmv", "cg jacobi", "cg jacobi", "ilu0", "ilu0", "ilut", "amg",
                       "amg", "vcycle", "batch", "ladder"])
    if kind == "spmv":
        if rng.random() < 0.4:
            return {"kind": "spmv", "problem": "ragged", "rows": log_int(2000, 600000),
                    "mean": rng.randint(7, 40)}
        return problem(["poisson", "varkappa", "convdiff"], {"kind": "spmv", "side": log_int(40, 2048)})
    if kind == "cg jacobi":
        return problem(["poisson", "varkappa"], {
            "kind": "solve", "solver": "CG", "precond": "JACOBI", "side": log_int(40, 720),
            "tol": rng.choice([1e-8, 1e-10]), "mixed": rng.random() < 0.25,
            "host": rng.random() < 0.5})
    if kind == "ilu0":
        return {"kind": "solve", "solver": "FGMRES", "precond": "ILU", "problem": "convdiff",
                "peclet": round(math.exp(rng.uniform(0.0, math.log(100.0))), 3),
                "side": log_int(60, 600), "tol": 1e-8, "mixed": False, "host": rng.random() < 0.5,
                "drop_tol": 0.0, "restart": 30}
    if kind == "ilut":
        return {"kind": "solve", "solver": "FGMRES", "precond": "ILU", "problem": "convdiff",
                "peclet": round(rng.uniform(0.05, 0.3), 3), "side": log_int(50, 180), "tol": 1e-8,
                "mixed": False, "host": rng.random() < 0.5, "drop_tol": 1e-4, "restart": 50}
    if kind == "amg":
        mixed = rng.random() < 0.5
        return problem(["poisson", "varkappa"], {
            "kind": "solve", "solver": "CG", "precond": "AMG",
            "side": log_int(150, 1500) if mixed else log_int(60, 260), "tol": 1e-10,
            "mixed": mixed, "host": rng.random() < 0.5, "cut": mixed})
    if kind == "vcycle":
        return problem(["poisson", "varkappa"], {"kind": "vcycle", "side": log_int(100, 1024)})
    if kind == "batch":
        lo = rng.randint(12, 40)
        return {"kind": "batch", "systems": log_int(30, 384), "lo": lo, "hi": lo + rng.randint(10, 80)}
    return problem(["convdiff", "varkappa", "helmholtz"], {
        "kind": "ladder", "side": log_int(32, 256), "tol": 1e-10, "mixed": True,
        "host": rng.random() < 0.5})


# ------------------------------------------------------------------------------ the inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _stencil(problem, n, seed, case):
    """(north, west, diag, east, south) of a 5-point operator on an n x n grid, as n x n
    arrays of the matrix entries; entries that leave the grid are zero."""
    full = lambda a: torch.full((n, n), float(a), dtype=F64, device="cuda")  # noqa: E731
    if problem in ("poisson", "helmholtz"):
        north = west = east = south = full(-1.0)
        diag = full(4.0)
        if problem == "helmholtz":      # c log-uniform, set by the seed
            u = random.Random(int(seed)).random()
            diag = diag + 0.1 * 100.0 ** u
    elif problem == "varkappa":         # lognormal per cell, harmonic face averages
        kap = torch.exp(case.get("sigma", 1.0) * torch.randn(n, n, dtype=F64, device="cuda",
                                                             generator=_gen(seed, 1)))
        fx = 2.0 * kap[:, :-1] * kap[:, 1:] / (kap[:, :-1] + kap[:, 1:])
        fy = 2.0 * kap[:-1] * kap[1:] / (kap[:-1] + kap[1:])
        west = -torch.cat([kap[:, :1], fx], 1)
        east = -torch.cat([fx, kap[:, -1:]], 1)
        north = -torch.cat([kap[:1], fy], 0)
        south = -torch.cat([fy, kap[-1:]], 0)
        diag = -(((north + west) + east) + south)
    else:                               # upwind convection-diffusion, wind at 30 degrees
        h = 1.0 / (n + 1)
        w = 2.0 * case["peclet"] * (n + 1)
        e, bx, by = 1.0 / (h * h), w * math.cos(math.pi / 6) / (2 * h), w * math.sin(math.pi / 6) / (2 * h)
        west, east, north, south = full(-e), full(-e - bx), full(-e), full(-e - by)
        diag = full(4.0 * e)
        diag[:, :-1] += bx
        diag[:-1] += by
        # some heterogeneity from the seed, so that no two systems are alike
        diag = diag * (1.0 + 0.05 * torch.rand(n, n, dtype=F64, device="cuda", generator=_gen(seed, 2)))
    north, west, east, south = (t.clone() for t in (north, west, east, south))
    north[0] = 0.0
    west[:, 0] = 0.0
    east[:, -1] = 0.0
    south[-1] = 0.0
    return north, west, diag, east, south


def _csr(st):
    """(row_ptr, col_idx, values) on the host of a stencil; columns sorted."""
    n = st[2].shape[0]
    node = torch.arange(n * n, device="cuda").view(n, n)
    i, j = node // n, node % n
    has = torch.stack([i > 0, j > 0, node >= 0, j < n - 1, i < n - 1], -1).view(-1, 5)
    col = torch.stack([node - n, node - 1, node, node + 1, node + n], -1).view(-1, 5)
    rp = torch.zeros(n * n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(has.sum(1), 0)
    v = torch.stack(st, -1).view(-1, 5)
    return (rp.int().cpu().numpy(), col[has].int().cpu().numpy(), v[has].cpu().numpy())


def _ragged(case, seed):
    """Unstructured CSR on the device (row_ptr, col_idx, values): row lengths geometric
    with the case's mean (1 to ~6 times it), columns within a band around the diagonal."""
    n, mean = case["rows"], case["mean"]
    g = _gen(seed, 3)
    u = torch.rand(n, dtype=F64, device="cuda", generator=g)
    length = (1 - mean * torch.log1p(-u)).clamp(1, 6 * mean).long()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), length)
    band = min(n - 1, 2000)
    off = (torch.randn(row.numel(), dtype=F64, device="cuda", generator=g) * band / 3).long()
    key = torch.unique(row * n + (row + off) % n)        # sorted, duplicates merged
    row, ci = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    v = torch.randn(key.numel(), dtype=F64, device="cuda", generator=g)
    return rp, ci, v


def _rhs(case, n, seed):
    lo = -1.0 if case.get("precond") == "AMG" or case["kind"] == "vcycle" else 0.0
    return lo + (1.0 - lo) * torch.rand(n, dtype=F64, device="cuda", generator=_gen(seed, 4))


def _params(case):
    over = {"tol": case.get("tol", 1e-8), "max_iter": 8000, "precision": 1 if case.get("mixed") else 0}
    if case["kind"] == "ladder":
        over.update(max_iter=4000, restart_size=30, drop_tol=0.0, ladder_mode=3)
    if "drop_tol" in case:
        over.update(drop_tol=case["drop_tol"], restart_size=case["restart"])
    if case.get("cut") or case["kind"] == "ladder":
        over.update(amg_omega=2.0 / 3.0, amg_coarse_limit=512, amg_levels=25, amg_stall_ratio=0.75)
    return H.SolverParams(**over)


def _batch_systems(case, seed):
    """(stencils, sides): even systems variable coefficients, odd ones convection."""
    r = random.Random(7)
    out = []
    for k in range(case["systems"]):
        side = r.randint(case["lo"], case["hi"])
        pe = math.exp(r.uniform(0.0, math.log(100.0)))
        out.append(_stencil("convdiff" if k % 2 else "varkappa", side, seed * 4099 + k,
                            {"peclet": pe, "sigma": 0.5}))
    return out


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "batch":
        sts = _batch_systems(case, seed)
        sol = [H.SOLVER_FGMRES if k % 2 else H.SOLVER_CG for k in range(len(sts))]
        pre = [H.PREC_ILU if k % 2 else H.PREC_JACOBI for k in range(len(sts))]
        p = H.SolverParams(tol=1e-8, max_iter=4000, restart_size=20, drop_tol=0.0)
        s["solver"] = B.BatchSolver([_csr(t) for t in sts], sol, pre, p)
        s["b"] = _rhs(case, s["solver"].N, seed).cpu().numpy()
        return s
    if case["problem"] == "ragged":
        n = case["rows"]
        rp, ci, v = _ragged(case, seed)
        csr = rp.int().cpu().numpy(), ci.int().cpu().numpy(), v.cpu().numpy()
    else:
        n = case["side"] ** 2
        csr = _csr(_stencil(case["problem"], case["side"], seed, case))
    s["A"] = H.SparseMatrix(n, n, *csr)
    # tensors the engine writes are made on its own stream, so that it sees them in order
    s["stream"] = torch.cuda.ExternalStream(s["A"].ctx.stream())
    b = _rhs(case, n, seed)
    s["b"] = b.cpu().numpy() if case.get("host") else b
    s["n"] = n
    if case["kind"] in ("solve", "ladder"):
        s["params"] = _params(case)
    if case["kind"] == "vcycle":
        s["M"] = H.AMGPreconditioner(amg_omega=2.0 / 3.0, amg_coarse_limit=512, amg_levels=25,
                                     amg_stall_ratio=0.75)
        s["M"].setup(s["A"])
    if case["kind"] in ("spmv", "vcycle"):
        s["y"] = torch.zeros(n, dtype=F64, device="cuda")
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------------------- one pass
def _x0(s):
    if s["case"].get("host"):
        return np.zeros(s["n"])
    with torch.cuda.stream(s["stream"]):
        return torch.zeros(s["n"], dtype=F64, device="cuda")


def run(s):
    kind = s["case"]["kind"]
    if kind == "spmv":
        return {"y": s["A"].spmv(s["b"], s["y"])}
    if kind == "vcycle":
        return {"z": s["M"].apply(s["b"], s["y"])}
    if kind == "batch":
        x, _, _ = s["solver"].solve(s["b"])
        return {"x": x}
    x = _x0(s)
    if kind == "ladder":
        H.AdaptiveSelector(s["params"]).solve(s["A"], s["b"], x)
        return {"x": x}
    c = s["case"]
    solver, _ = H.SolverFactory.make(c["solver"], c["precond"], s["A"], s["params"])
    solver.solve(s["A"], s["b"], x)
    return {"x": x}


def work(case):
    """The matrix and the right-hand side (or multiplied vector) read once, the result
    written once; two operations an entry."""
    if case["kind"] == "batch":
        r = random.Random(7)
        n = nnz = 0
        for _ in range(case["systems"]):
            side = r.randint(case["lo"], case["hi"])
            r.random()
            n += side * side
            nnz += 5 * side * side - 4 * side
    elif case["problem"] == "ragged":
        n = case["rows"]
        nnz = n * case["mean"]
    else:
        n = case["side"] ** 2
        nnz = 5 * n - 4 * case["side"]
    return {"bytes": 4 * (n + 1) + 12 * nnz + 16 * n, "flops": 2 * nnz}


# ------------------------------------------------------------------------ 64-bit reference
def _mul(st, x):
    north, west, diag, east, south = st
    y = diag * x
    y[1:] += north[1:] * x[:-1]
    y[:, 1:] += west[:, 1:] * x[:, :-1]
    y[:, :-1] += east[:, :-1] * x[:, 1:]
    y[:-1] += south[:-1] * x[1:]
    return y


def _cg(st, b):
    """Conjugate gradients with diagonal scaling, its residual replaced by the true one."""
    x = torch.zeros_like(b)
    target = 1e-14 * float(b.norm())
    for _ in range(3):
        r = b - _mul(st, x)
        z = r / st[2]
        p = z.clone()
        rho = (r * z).sum()
        for k in range(20000):
            q = _mul(st, p)
            a = rho / (p * q).sum()
            x += a * p
            r -= a * q
            z = r / st[2]
            new = (r * z).sum()
            p = z + (new / rho) * p
            rho = new
            if k % 50 == 49 and float(r.norm()) < target:
                break
    return x


def _direct(sts, bs):
    """Block tridiagonal elimination over grid rows, all systems at once (smaller grids
    padded with identity rows), and one step of refinement."""
    m = max(t[2].shape[0] for t in sts)
    pad = lambda a, fill: torch.nn.functional.pad(a, (0, m - a.shape[1], 0, m - a.shape[0]), value=fill)  # noqa: E731
    north, west, diag, east, south = (
        torch.stack([pad(t[k], 1.0 if k == 2 else 0.0) for t in sts]) for k in range(5))
    inv = []
    for i in range(m):
        d = torch.diag_embed(diag[:, i]) + torch.diag_embed(west[:, i, 1:], -1) + torch.diag_embed(east[:, i, :-1], 1)
        if i:
            d = d - north[:, i, :, None] * inv[-1] * south[:, i - 1, None, :]
        inv.append(torch.linalg.inv(d))

    def solve(b):
        y = []
        for i in range(m):
            r = b[:, i] - (north[:, i] * y[-1] if i else 0.0)
            y.append((inv[i] @ r[:, :, None])[:, :, 0])
        for i in range(m - 2, -1, -1):
            y[i] = y[i] - (inv[i] @ (south[:, i] * y[i + 1])[:, :, None])[:, :, 0]
        return torch.stack(y, 1)

    b = torch.stack([pad(v, 0.0) for v in bs])
    x = solve(b)
    full = (north, west, diag, east, south)
    r = torch.stack([b[k] - _mul([c[k] for c in full], x[k]) for k in range(len(sts))])
    x = x + solve(r)
    return [x[k, :t[2].shape[0], :t[2].shape[0]].reshape(-1) for k, t in enumerate(sts)]


def exact(case, seed):
    if case["kind"] == "vcycle":
        return None                     # the hierarchy is the engine's own
    if case["kind"] == "batch":
        sts = _batch_systems(case, seed)
        sides = [t[2].shape[0] for t in sts]
        b = _rhs(case, sum(k * k for k in sides), seed)
        bs = [v.view(k, k) for v, k in zip(b.split([k * k for k in sides]), sides)]
        return {"x": torch.cat(_direct(sts, bs))}
    if case["problem"] == "ragged":
        rp, ci, v = _ragged(case, seed)
        x = _rhs(case, case["rows"], seed)
        row = torch.repeat_interleave(torch.arange(case["rows"], device="cuda"), rp[1:] - rp[:-1])
        return {"y": torch.zeros_like(x).index_add_(0, row, v * x[ci])}
    n = case["side"]
    st = _stencil(case["problem"], n, seed, case)
    b = _rhs(case, n * n, seed).view(n, n)
    if case["kind"] == "spmv":
        return {"y": _mul(st, b).view(-1)}
    if case["problem"] == "convdiff":
        return {"x": _direct([st], [b])[0]}
    return {"x": _cg(st, b).view(-1)}
