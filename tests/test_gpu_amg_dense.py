"""The dense ends of the AMG setup (-m gpu): the coarsest level's factorisation, inverse and
solve at the sizes where they change form, and Galerkin products of near-dense levels
(window columns beyond one pass of 256, left rows beyond the 256 staged), against the oracle.
"""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P
from hsps_b200._abi import default_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def csr(D):
    r, c = np.nonzero(D)
    rp = np.zeros(len(D) + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=len(D)))
    return rp, c.astype(np.int32), D[r, c].copy()


def one_level(A, n):
    M = H.AMGPreconditioner(amg_coarse_limit=n)
    M.setup(H.SparseMatrix(n, n, *A))
    assert M.levels() == 1
    return M


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 95, 96])
def test_coarse_elimination_bitwise(orc, n):
    # rows in random order: the diagonal is small and most steps interchange rows
    rng = np.random.default_rng(n)
    D = (rng.standard_normal((n, n)) + 3.0 * n * np.eye(n))[rng.permutation(n)]
    D[rng.random((n, n)) < 0.2] *= 0.0
    D += 1e-3 * np.eye(n)
    A = csr(D)
    r = rng.standard_normal(n)
    z = one_level(A, n).apply(r)
    assert np.array_equal(z, orc.amg_apply(*A, r, default_params(amg_coarse_limit=n)))


def test_coarse_elimination_skips_empty_columns_bitwise(orc):
    rng = np.random.default_rng(5)
    D = rng.standard_normal((40, 40)) + 10.0 * np.eye(40)
    D[:, 7] = 0.0
    D[7, 7] = 1e-20                      # below the pivot threshold
    D[:, 23] = 0.0
    D[3, 23] = 1e-15
    A = csr(D)
    r = rng.standard_normal(40)
    z = one_level(A, 40).apply(r)
    assert np.array_equal(z, orc.amg_apply(*A, r, default_params(amg_coarse_limit=40)))


@pytest.mark.parametrize("n", [97, 155, 256, 511, 800, 1024])
def test_coarse_inverse(n):
    # an explicit inverse: the residual of a well-conditioned system (condition number ~4)
    # stays within n * 1e-16 * 4 of the right-hand side; 1e-11 leaves a factor of 25 at 1,024
    rng = np.random.default_rng(n)
    D = (rng.standard_normal((n, n)) / np.sqrt(n) + 3.0 * np.eye(n))[rng.permutation(n)]
    r = rng.standard_normal(n)
    z = one_level(csr(D), n).apply(r)
    assert np.linalg.norm(r - D @ z) <= 1e-11 * np.linalg.norm(r)


@pytest.mark.parametrize("n", [1025, 1087, 1088, 1089, 1279, 1281, 1345, 2305])
@pytest.mark.parametrize("shuffled", [False, True])
def test_coarse_inverse_blocked(n, shuffled):
    # beyond 1,024 rows: blocks of 64 in groups of 256.  With its diagonal in place D needs
    # no interchanges (the same bound, a factor of 10 at 2,305); shuffled, with zeros on the
    # diagonal that end the attempt without them, it takes the pivoted form.
    rng = np.random.default_rng(n)
    D = rng.standard_normal((n, n)) / np.sqrt(n) + 3.0 * np.eye(n)
    if shuffled:
        D = D[rng.permutation(n)]
        D[np.arange(0, n, 7), np.arange(0, n, 7)] = 0.0
    r = rng.standard_normal(n)
    z = one_level(csr(D), n).apply(r)
    assert np.linalg.norm(r - D @ z) <= 1e-11 * np.linalg.norm(r)


def near_dense(n, per_row, seed):
    rng = np.random.default_rng(seed)
    D = np.where(rng.random((n, n)) < per_row / n, -rng.random((n, n)), 0.0)
    D = np.triu(D, 1)
    D = D + D.T
    np.fill_diagonal(D, 0.3 - D.sum(1))
    return csr(D)


@pytest.mark.parametrize("name,A", [
    ("dense_300", near_dense(300, 300, 1)),
    ("dense_620", near_dense(620, 620, 2)),
    ("half_dense_700", near_dense(700, 350, 3)),
    ("rows_100_of_1500", near_dense(1500, 100, 4)),
    ("grid_60", P.varkappa_poisson_2d(60, 1.0, 5)),
], ids=lambda a: a if isinstance(a, str) else "")
@pytest.mark.parametrize("theta", [0.25, 0.9])
def test_hierarchy_bitwise(orc, name, A, theta):
    n = len(A[0]) - 1
    M = H.AMGPreconditioner(amg_strong=theta)
    M.setup(H.SparseMatrix(n, n, *A))
    ref = orc.amg_hierarchy(*A, default_params(amg_strong=theta))
    assert M.levels() == len(ref)
    for l in range(M.levels()):
        for which, key in ((0, "A"), (1, "P"), (2, "R")):
            if which and l == M.levels() - 1:
                continue
            got, want = M.level_matrix(l, which), ref[l][key]
            assert got[:2] == want[:2]
            for x, y in zip(got[2:], want[2:]):
                assert np.array_equal(x, y), (l, key)
