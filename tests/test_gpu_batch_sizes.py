"""Batched systems at the edges of the scheduling groups (100, 200, 640, 1,024, 4,096, 16,384
rows) and above the last, where the vectors stay in global memory, each method (-m gpu).

A system's solution is compared with a direct solve of it (scipy's sparse LU in FP64): both have
a relative residual of at most 1e-10, and the systems' condition numbers, at most 2e4 here,
carry that to a relative error below 4e-6."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix
from scipy.sparse.linalg import splu

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import batch as B
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def chain(n, seed, sym):
    """Banded operator with offsets 1 and 7, diagonally dominant; symmetric or not."""
    rng = np.random.default_rng(seed)
    r, c, v = [np.arange(n)], [np.arange(n)], [4.0 + rng.uniform(0.05, 0.5, n)]
    for o in (1, 7):
        i = np.arange(max(0, n - o))
        w = -rng.uniform(0.5, 1.0, len(i))
        r += [i, i + o]
        c += [i + o, i]
        v += [w, w if sym else 0.4 * w]
    r, c, v = map(np.concatenate, (r, c, v))
    k = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.bincount(r, minlength=n)
    return np.cumsum(rp).astype(np.int32), c[k].astype(np.int32), v[k]


SIZES = [1, 2, 31, 32, 33, 99, 100, 101, 199, 200, 201, 639, 640, 641, 1023, 1024, 1025, 4096, 4097, 16384, 16385,
         20011]


@pytest.mark.parametrize("solver,precond", [("CG", "JACOBI"), ("CG", "NONE"), ("FGMRES", "ILU"), ("FGMRES", "JACOBI")])
def test_every_group_against_a_direct_solve(solver, precond):
    systems = [chain(n, n, solver == "CG") for n in SIZES]
    rhs = [P.rhs(n, 3 + n, -1.0, 1.0) for n in SIZES]
    p = H.SolverParams(tol=1e-10, max_iter=4000, restart_size=20, drop_tol=0.0)
    s = getattr(H, "SOLVER_" + solver)
    pc = getattr(H, "PREC_" + precond)
    bs = B.BatchSolver(systems, s, pc, p)
    x, res, _ = bs.solve(rhs)
    for n, A, b, xk, o in zip(SIZES, systems, rhs, bs.split(x), res):
        assert o["status"] == 0 and o["converged"] == 1, (n, o)
        M = csr_matrix((A[2], A[1], A[0]), shape=(n, n))
        assert np.linalg.norm(b - M @ xk) <= 1.001e-10 * np.linalg.norm(b), n
        want = splu(M.tocsc()).solve(b)
        assert np.linalg.norm(xk - want) <= 4e-6 * np.linalg.norm(want), n
    # alone: the same bits, whatever else the batch holds
    for k in (4, 6, 7, 10, 13, 20):
        one = B.BatchSolver([systems[k]], s, pc, p)
        x1, r1, _ = one.solve([rhs[k]])
        one.release()
        assert r1[0]["iterations"] == res[k]["iterations"] and np.array_equal(x1, bs.split(x)[k]), SIZES[k]
    bs.release()


@pytest.mark.parametrize("side", [100, 129, 150])
def test_grid_ilu_against_a_direct_solve(side):
    # the elimination's levels: 10,000 rows (shared vector), 16,641 and 22,500 (global memory)
    A = P.convection_diffusion_2d(side, 1.0, *P.convdiff_wind(side, 3.0))
    n = side * side
    b = P.rhs(n, 5)
    p = H.SolverParams(tol=1e-10, max_iter=4000, restart_size=20, drop_tol=0.0)
    bs = B.BatchSolver([A], H.SOLVER_FGMRES, H.PREC_ILU, p)
    x, res, _ = bs.solve([b])
    bs.release()
    M = csr_matrix((A[2], A[1], A[0]), shape=(n, n))
    want = splu(M.tocsc()).solve(b)
    assert res[0]["converged"] == 1
    assert np.linalg.norm(x - want) <= 4e-6 * np.linalg.norm(want)


def test_many_small_systems_all_solved():
    # more than one round of tickets for every warp of the chip
    systems = [chain(20 + k % 80, k, k % 2 == 0) for k in range(5000)]
    rhs = [P.rhs(len(a[0]) - 1, k) for k, a in enumerate(systems)]
    so = [H.SOLVER_CG if k % 2 == 0 else H.SOLVER_FGMRES for k in range(5000)]
    pr = [H.PREC_JACOBI if k % 2 == 0 else H.PREC_ILU for k in range(5000)]
    bs = B.BatchSolver(systems, so, pr, H.SolverParams(tol=1e-10, max_iter=4000, restart_size=20, drop_tol=0.0))
    x, res, _ = bs.solve(rhs)
    assert all(o["converged"] == 1 for o in res)
    for k in range(0, 5000, 97):
        A, n = systems[k], len(rhs[k])
        M = csr_matrix((A[2], A[1], A[0]), shape=(n, n))
        assert np.linalg.norm(rhs[k] - M @ bs.split(x)[k]) <= 1.001e-10 * np.linalg.norm(rhs[k])
    bs.release()
