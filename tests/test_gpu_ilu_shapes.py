"""ILU(0) on triangles of every shape its kernels tell apart, bit for bit against the
oracle: level sets, factor values and apply (-m gpu).  The shapes sit at the edges of the
sweep kernels' ring (4,096 solution values), entry places (2, 4, 8, 16 a row) and steps (up
to 864 rows), of the elimination's short rows (8 entries) and of the level kernel's row
blocks (1,024).
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


def from_offsets(n, offs, seed, keep=1.0):
    """CSR with entries at i + o (o in offs, each kept with probability `keep`) and a
    dominant diagonal."""
    rng = np.random.default_rng(seed)
    r, c = [np.arange(n)], [np.arange(n)]
    for o in offs:
        i = np.arange(max(0, -o), min(n, n - o))
        i = i[rng.random(len(i)) < keep]
        r.append(i)
        c.append(i + o)
    r, c = np.concatenate(r), np.concatenate(c)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    v = rng.uniform(-1.0, 1.0, len(r))
    v[r == c] = len(offs) + rng.uniform(0.5, 1.5, n)
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, r + 1, 1)
    return np.cumsum(rp).astype(np.int32), c.astype(np.int32), v


SHAPES = [
    ("one_row", lambda: from_offsets(1, [], 0)),
    ("diagonal_only", lambda: from_offsets(777, [], 1)),
    ("tridiagonal_5000", lambda: from_offsets(5000, [-1, 1], 2)),          # 5,000 levels of one row
    ("tridiagonal_1024", lambda: from_offsets(1024, [-1, 1], 3)),          # one row block exactly
    ("tridiagonal_1025", lambda: from_offsets(1025, [-1, 1], 4)),
    ("far_entries", lambda: from_offsets(8200, [-6000, -4097, -4096, -4095, -1, 1, 4096, 6000], 5)),
    ("wide_steps_1500", lambda: from_offsets(9000, [-1500, 1500], 6)),     # two steps a level
    ("wide_steps_865", lambda: from_offsets(4000, [-865, 865], 7)),
    ("wide_864_long", lambda: from_offsets(4100, [-864 - k for k in range(6)] + [864, 865], 8)),
    ("grid_73", lambda: P.varkappa_poisson_2d(73, 1.0, 9)),
    ("band_20", lambda: from_offsets(3000, list(range(-20, 0)) + list(range(1, 12)), 10)),
    ("rows_16_17", lambda: from_offsets(900, list(range(-16, 0)) + list(range(1, 18)), 11)),
    ("rows_17_16", lambda: from_offsets(900, list(range(-17, 0)) + list(range(1, 17)), 12)),
    ("rows_9_8", lambda: from_offsets(2100, [-300 - 7 * k for k in range(9)] + [256 + 5 * k for k in range(8)], 19)),
    ("rows_5_4", lambda: from_offsets(5000, [-577 - k for k in range(5)] + [576, 580, 700, 900], 20)),
    ("rows_3_2", lambda: from_offsets(5000, [-1, -2, -900, 1, 900], 21)),
    ("gaps", lambda: from_offsets(7000, [-130, -64, -33, -1, 1, 33, 64, 130], 13, 0.6)),
    ("two_chains", lambda: from_offsets(6000, [-2, 2], 14)),               # level kernel gives up
    ("many_chains", lambda: from_offsets(3000, [-7, -5, -3, 2, 4, 9], 15)),
    ("lower_wide_upper_chain", lambda: from_offsets(6000, [1, 2], 16)),
    ("upper_wide_lower_chain", lambda: from_offsets(6000, [-1], 17)),
    ("both_wide", lambda: from_offsets(20000, [-10000, 10000], 18)),
]


@pytest.mark.parametrize("name,make", SHAPES, ids=[s[0] for s in SHAPES])
def test_ilu0_shapes_bitwise(orc, name, make):
    A = make()
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    I = H.ILUPreconditioner()
    I.setup(M)
    for which in (0, 1):
        nd, ld = I.level_sets(which)
        no, lo = orc.levels(A[0], A[1], which)
        assert nd == no and np.array_equal(ld, lo)
    rc, lu = orc.ilu0(*A)
    assert rc == 0
    assert np.array_equal(I.factors(), lu)
    for seed in (31, 32):
        r = P.rhs(n, seed, -1.0, 1.0)
        rc, z = orc.ilu_apply(A[0], A[1], lu, r)
        assert rc == 0 and np.array_equal(I.apply(r), z)


@pytest.mark.parametrize("name", ["tridiagonal_5000", "far_entries", "wide_steps_1500", "band_20",
                                  "rows_17_16", "lower_wide_upper_chain", "both_wide"])
def test_ilu0_shapes_fp32(orc, name):
    # the FP32 sweeps, inside a mixed-precision FGMRES solve certified in FP64
    A = dict((s[0], s[1]) for s in SHAPES)[name]()
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    s, _ = H.SolverFactory.make("FGMRES", "ILU", M, H.SolverParams(tol=1e-10, drop_tol=0.0, precision=1,
                                                                  restart_size=30))
    b, x = P.rhs(n, 5, -1.0, 1.0), np.zeros(n)
    assert s.solve(M, b, x)
    r = b - orc.spmv(*A, x)
    assert np.linalg.norm(r) <= 1.05e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("n,off,zero", [(5000, 1, [0]), (5000, 1, [4998]), (5000, 1, [3, 2047, 4000]),
                                        (9000, 1500, [1499]), (9000, 700, [20, 8290]), (9000, 5000, [17, 3900])])
def test_ilu0_vanishing_pivot(orc, n, off, zero):
    # rows i and i + off: a pivot that is exactly 0 where row i + off eliminates with it; the
    # first such pivot in index order is reported
    rp, ci, v = from_offsets(n, [-off, off], 40)
    row = np.repeat(np.arange(n), np.diff(rp))
    v[row == ci] = 4.0
    v[row != ci] = -1.0
    for z in zero:
        v[(row == z) & (ci != z)] = 0.0
        v[(row == z) & (ci == z)] = 0.0
    assert orc.ilu0(rp, ci, v)[0] == H._abi.ERR_ZERO_PIVOT
    M = H.SparseMatrix(n, n, rp, ci, v)
    with pytest.raises(H.HamlssError) as e:
        H.ILUPreconditioner().setup(M)
    assert e.value.code == H._abi.ERR_ZERO_PIVOT
    assert str(e.value).rstrip().endswith("row %d" % min(zero))
    v[row == ci] = 4.0                                     # and the same pattern factors again
    M = H.SparseMatrix(n, n, rp, ci, v)
    I = H.ILUPreconditioner()
    I.setup(M)
    assert np.array_equal(I.factors(), orc.ilu0(rp, ci, v)[1])
