"""The persistent CG iteration at the edges of its shapes (-m gpu): rows a block (256 to
3,584; 1 to 7 a thread), one cluster or the whole grid, the most rows it holds, windows
and entries that do not fit (the two-launch iteration), and its stop rules.

A fixed number of trips K is compared with the oracle's iterates: the two differ by the
order of the dot products, a relative 1e-16 or so a trip that CG amplifies little before
convergence; 1e-11 after 10 trips leaves a margin of four digits.
"""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def banded(n, offs, seed):
    """Symmetric, diagonally dominant CSR with entries at +-offs; rows of uneven length."""
    rng = np.random.default_rng(seed)
    r, c, v = [np.arange(n)], [np.arange(n)], [2.05 * len(offs) + rng.uniform(0, 1, n)]
    for o in offs:
        i = np.arange(n - o) if n > o else np.arange(0)
        i = i[rng.random(len(i)) < 0.9]
        w = -rng.uniform(0.2, 1.0, len(i))
        r += [i, i + o]
        c += [i + o, i]
        v += [w, w]
    r, c, v = map(np.concatenate, (r, c, v))
    order = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, r + 1, 1)
    return np.cumsum(rp).astype(np.int32), c[order].astype(np.int32), v[order]


def run(A, precond, b, x0, **over):
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    s, _ = H.SolverFactory.make("CG", precond, M, H.SolverParams(**over))
    x, st = x0.copy(), H.SolverStats()
    ok = s.solve(M, b, x, st)
    return ok, x, st


SIZES = [255, 256, 257, 4096, 4097, 8193, 16385, 28672, 28673, 37889, 75777, 151553, 303105, 500001, 530433]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
def test_fixed_trips(orc, n, precond):
    A = banded(n, [1, 37] if n > 40 else [1], n)
    b = P.rhs(n, 3, -1.0, 1.0)
    x0 = P.rhs(n, 4, -1.0, 1.0)
    K = 10
    over = dict(tol=1e-300, max_iter=K)
    ok, x, st = run(A, precond, b, x0, **over)
    rc, xo, so = orc.solve(0, 1 if precond == "JACOBI" else 0, *A, b, x0=x0, params=H.SolverParams(**over))
    assert not ok and st.iterations == so.iterations
    assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)
    assert abs(st.final_residual - so.final_residual) <= 1e-9 * so.final_residual


@pytest.mark.parametrize("n", [1, 2, 3])
def test_tiny(orc, n):
    A = banded(n, [1], n)
    b = P.rhs(n, 3, -1.0, 1.0)
    over = dict(tol=1e-8, max_iter=10)
    ok, x, st = run(A, "JACOBI", b, np.zeros(n), **over)
    rc, xo, so = orc.solve(0, 1, *A, b, params=H.SolverParams(**over))
    assert ok and st.iterations == so.iterations
    assert np.linalg.norm(x - xo) <= 1e-14 * np.linalg.norm(xo)


@pytest.mark.parametrize("name,A", [
    ("window_too_wide", banded(60000, [1, 29990], 1)),          # a block spans most columns
    ("wide_window", banded(30000, [1, 9000], 2)),
    ("many_entries", banded(20000, list(range(1, 34)), 3)),     # ~60 entries a row
    ("too_many_entries", banded(90000, list(range(1, 21)), 4)),
    ("varkappa_200", P.varkappa_poisson_2d(200, 1.0, 5)),
], ids=lambda a: a if isinstance(a, str) else "")
def test_converges_like_the_oracle(orc, name, A):
    n = len(A[0]) - 1
    b = P.rhs(n, 6)
    over = dict(tol=1e-9, max_iter=4000)
    ok, x, st = run(A, "JACOBI", b, np.zeros(n), **over)
    rc, xo, so = orc.solve(0, 1, *A, b, params=H.SolverParams(**over))
    assert ok and so.converged and abs(st.iterations - so.iterations) <= 1
    assert st.true_residual <= 2e-9


def test_more_trips_than_a_launch_holds():
    # 4,096 trips a launch: the state travels through memory between launches
    A = P.varkappa_poisson_2d(64, 3.5, 1)
    n = 64 * 64
    b = P.rhs(n, 2, -1.0, 1.0)
    ok, x, st = run(A, "NONE", b, np.zeros(n), tol=1e-300, max_iter=4700)
    assert not ok and st.iterations == 4700 and np.isfinite(x).all()


def test_repeatable():
    A = P.varkappa_poisson_2d(333, 1.0, 8)
    n = 333 * 333
    b = P.rhs(n, 9)
    runs = [run(A, "JACOBI", b, np.zeros(n), tol=1e-8, max_iter=4000) for _ in range(2)]
    assert runs[0][0] and np.array_equal(runs[0][1], runs[1][1])


def test_zero_rhs_and_exact_guess():
    A = P.poisson_2d(20)
    ok, x, st = run(A, "JACOBI", np.zeros(400), np.zeros(400), tol=1e-8, max_iter=100)
    assert ok and st.iterations == 0 and not x.any()
    xs = P.rhs(400, 1)
    M = H.SparseMatrix(400, 400, *A)
    ok, x, st = run(A, "JACOBI", M.spmv(xs), xs, tol=1e-8, max_iter=100)
    assert ok and st.iterations == 0 and np.array_equal(x, xs)


def test_nonfinite_is_an_error():
    A = P.poisson_2d(20)
    b = np.ones(400)
    b[7] = np.inf
    with pytest.raises(H.HamlssError) as e:
        run(A, "JACOBI", b, np.zeros(400), tol=1e-8, max_iter=100)
    assert e.value.code == H._abi.ERR_NONFINITE


@pytest.mark.parametrize("side,trips", [(20, 101), (64, 316), (150, 729), (200, 898), (420, 1992)])
def test_mixed_precision_updates(orc, side, trips):
    # the FP32 iteration leaves its launch for every FP64 residual update; `trips`: what the
    # two-launch form of the same scheme takes (measured), which differs by summation order
    A = P.varkappa_poisson_2d(side, 1.0, side)
    n = side * side
    b = P.rhs(n, 3, -1.0, 1.0)
    ok, x, st = run(A, "JACOBI", b, np.zeros(n), tol=1e-10, max_iter=8000, precision=1)
    assert ok and st.outer_iterations >= 2 and st.true_residual <= 1e-10
    assert abs(st.iterations - trips) <= 1
    r = b - orc.spmv(*A, x)
    assert np.linalg.norm(r) <= 1.001e-10 * np.linalg.norm(b)
