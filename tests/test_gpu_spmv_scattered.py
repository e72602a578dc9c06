"""FP64 products of short-row operators whose neighbouring rows' columns lie apart: the form
of the bulk-copy kernel that has a row's gathers in flight together, bit for bit against the
plain loop, and the operators on the other side of that rule (-m gpu)."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def permuted(A, seed):
    rp, ci, v = A
    n = len(rp) - 1
    p = np.random.default_rng(seed).permutation(n)
    r, c = p[np.repeat(np.arange(n), np.diff(rp))], p[ci]
    o = np.lexsort((c, r))
    out = np.zeros(n + 1, np.int64)
    out[1:] = np.bincount(r, minlength=n)
    return np.cumsum(out).astype(np.int32), c[o].astype(np.int32), v[o]


def random_rows(n, lengths, seed, band=None):
    """CSR with about `lengths` random columns a row (duplicates merged), in a band or anywhere."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), lengths)
    c = rng.integers(0, n, len(r)) if band is None else np.clip(r + rng.integers(-band, band + 1, len(r)), 0, n - 1)
    key = np.unique(r * np.int64(n) + c)
    r, c = key // n, key % n
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.bincount(r, minlength=n)
    return np.cumsum(rp).astype(np.int32), c.astype(np.int32), rng.standard_normal(len(r))


def long_tiles(n):
    """Rows of 3 with some tiles of 9: more entries than a stage holds."""
    out = np.full(n, 3)
    out[5000:5600] = 9
    out[n - 100:] = 9
    return out


CASES = {
    "grid_permuted": lambda: permuted(P.varkappa_poisson_2d(200, 1.0, 1), 2),
    "grid_32768": lambda: permuted(P.varkappa_poisson_2d(182, 1.0, 1), 3),        # 33,124 rows
    "smallest": lambda: random_rows(32768, np.full(32768, 4), 4),
    "one_less": lambda: random_rows(32767, np.full(32767, 4), 4),                 # the plain kernel
    "lengths_0_to_9": lambda: random_rows(40001, np.random.default_rng(5).integers(0, 10, 40001), 5),
    "band_100": lambda: random_rows(50003, np.full(50003, 4), 6, 100),
    "band_4": lambda: random_rows(50003, np.full(50003, 4), 7, 4),                # near: the other form
    "long_tiles": lambda: random_rows(60000, long_tiles(60000), 8),
    "mostly_empty": lambda: random_rows(70000, np.where(np.arange(70000) % 97 == 0, 40, 0), 9),
    "grid_natural": lambda: P.varkappa_poisson_2d(200, 1.0, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_bitwise(orc, name):
    A = CASES[name]()
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    for seed in (1, 2):
        x = P.rhs(n, seed, -1.0, 1.0)
        assert np.array_equal(M.spmv(x), orc.spmv(*A, x))


def test_skewed_rows_keep_their_split(orc):
    ln = np.full(50000, 3)
    ln[777] = 30000
    A = random_rows(50000, ln, 10)
    x = P.rhs(50000, 3, -1.0, 1.0)
    assert np.array_equal(H.SparseMatrix(50000, 50000, *A).spmv(x), orc.spmv(*A, x))


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
def test_cg_on_scattered_rows(orc, precond):
    # ten trips against the oracle's iterates (1e-11: the sums' order, four digits of margin);
    # too wide a window for the persistent iteration
    A = permuted(P.varkappa_poisson_2d(260, 0.5, 1), 4)
    n = len(A[0]) - 1
    b = P.rhs(n, 3, -1.0, 1.0)
    p = H.SolverParams(tol=1e-300, max_iter=10)
    M = H.SparseMatrix(n, n, *A)
    s, _ = H.SolverFactory.make("CG", precond, M, p)
    x = np.zeros(n)
    s.solve(M, b, x)
    rc, xo, so = orc.solve(0, 1 if precond == "JACOBI" else 0, *A, b, params=p)
    assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)
