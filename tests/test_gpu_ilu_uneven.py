"""ILU(0) on triangles whose rows are mostly much shorter than their longest: such triangles
leave the ring kernel, each for itself, and the results stay the oracle's bits (-m gpu)."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def with_rows(A, rows, cols):
    """A with extra entries (-0.01) at (rows, cols)."""
    rp, ci, v = A
    n = len(rp) - 1
    r = np.concatenate([np.repeat(np.arange(n), np.diff(rp)), rows])
    c, v = np.concatenate([ci, cols]), np.concatenate([v, np.full(len(rows), -0.01)])
    o = np.lexsort((c, r))
    out = np.zeros(n + 1, np.int64)
    out[1:] = np.bincount(r, minlength=n)
    return np.cumsum(out).astype(np.int32), c[o].astype(np.int32), v[o]


def banded(n, offs, keep, seed):
    rng = np.random.default_rng(seed)
    r, c = [np.arange(n)], [np.arange(n)]
    for o in offs:
        i = np.arange(max(0, -o), min(n, n - o))
        i = i[rng.random(len(i)) < keep]
        r.append(i)
        c.append(i + o)
    r, c = np.concatenate(r), np.concatenate(c)
    o = np.lexsort((c, r))
    r, c = r[o], c[o]
    v = rng.uniform(-1.0, 1.0, len(r))
    v[r == c] = len(offs) + rng.uniform(0.5, 1.5, n)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.bincount(r, minlength=n)
    return np.cumsum(rp).astype(np.int32), c.astype(np.int32), v


GRID = P.varkappa_poisson_2d(150, 1.0, 1)
N = 150 * 150
MID = N // 2
WIDE = [-1500 - 7 * k for k in range(16)]
CASES = {
    "lower_row_of_16": lambda: with_rows(GRID, np.full(14, MID), MID - 1000 - 37 * np.arange(14)),
    "upper_row_of_16": lambda: with_rows(GRID, np.full(14, MID), MID + 1000 + 37 * np.arange(14)),
    "both": lambda: with_rows(GRID, np.full(28, MID), np.r_[MID - 1000 - 37 * np.arange(14), MID + 1000 + 37 * np.arange(14)]),
    "lower_quarter_of_16": lambda: banded(30000, WIDE + [1500], 0.25, 2),
    "upper_quarter_of_16": lambda: banded(30000, [-w for w in WIDE] + [-1500], 0.25, 3),
    "quarter_of_8": lambda: banded(30000, WIDE[:8] + [-w for w in WIDE[:8]], 0.25, 4),
    "half_of_16": lambda: banded(24000, WIDE + [-w for w in WIDE], 0.5, 5),
}


@pytest.mark.parametrize("name", CASES)
def test_bitwise(orc, name):
    A = CASES[name]()
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    I = H.ILUPreconditioner()
    I.setup(M)
    rc, lu = orc.ilu0(*A)
    assert rc == 0 and np.array_equal(I.factors(), lu)
    for seed in (31, 32):
        r = P.rhs(n, seed, -1.0, 1.0)
        rc, z = orc.ilu_apply(A[0], A[1], lu, r)
        assert rc == 0 and np.array_equal(I.apply(r), z)


@pytest.mark.parametrize("name", ["lower_row_of_16", "upper_row_of_16", "half_of_16"])
def test_fp32_in_a_mixed_solve(orc, name):
    A = CASES[name]()
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    s, _ = H.SolverFactory.make("FGMRES", "ILU", M, H.SolverParams(tol=1e-10, drop_tol=0.0, precision=1,
                                                                  restart_size=30))
    b, x = P.rhs(n, 5, -1.0, 1.0), np.zeros(n)
    assert s.solve(M, b, x)
    assert np.linalg.norm(b - orc.spmv(*A, x)) <= 1.05e-10 * np.linalg.norm(b)
