"""FGMRES' multi-vector dots and updates at the edges of their shapes (-m gpu): vectors of
1 to 63 (the 4, 8, 16, 32 and 64 forms, whole and in part), lengths around a block's 256
entries and around the entries one pass of the grid covers (592 blocks).

After m steps of one cycle the iterate is the minimiser of the residual over the Krylov
space, whatever the order of its sums.  The dense least-squares solution in the same space,
formed in NumPy with a twice-orthogonalised basis, is the yardstick; the matrices are
strongly diagonally dominant, so the problem's condition number is below 1e2 and the two
differ by some 1e2 * m * 1e-16: 1e-11 relative is a margin of over two digits at m = 63.
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


def matrix(n):
    i = np.arange(n)
    r, c, v = [i], [i], [4.0 + 1.5 * np.sin(0.7 * i)]
    for o, w in ((1, -0.9), (-1, -0.6), (17, 0.5)):
        j = i[(i + o >= 0) & (i + o < n)]
        r.append(j)
        c.append(j + o)
        v.append(np.full(len(j), w))
    r, c, v = map(np.concatenate, (r, c, v))
    order = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, r + 1, 1)
    return np.cumsum(rp).astype(np.int32), c[order].astype(np.int32), v[order]


def krylov_minimiser(A, b, m):
    V, Hm = [b / np.linalg.norm(b)], np.zeros((m + 1, m))
    for j in range(m):
        w = A(V[j])
        for _ in range(2):
            h = np.array([u @ w for u in V])
            w = w - np.stack(V, 1) @ h
            Hm[:j + 1, j] += h
        Hm[j + 1, j] = np.linalg.norm(w)
        V.append(w / Hm[j + 1, j])
    e = np.zeros(m + 1)
    e[0] = np.linalg.norm(b)
    return np.stack(V[:m], 1) @ np.linalg.lstsq(Hm, e, rcond=None)[0]


@pytest.mark.parametrize("n,m", [(2, 1), (200, 3), (255, 4), (256, 5), (257, 8), (511, 9), (513, 12), (5000, 13),
                                 (5000, 20), (5000, 40), (32761, 20), (32761, 63), (151552, 12), (151553, 9), (303105, 17)])
def test_one_cycle(orc, n, m):
    csr = matrix(n)
    M = H.SparseMatrix(n, n, *csr)
    b = P.rhs(n, 6, -1.0, 1.0)
    want = krylov_minimiser(lambda x: orc.spmv(*csr, x), b, m)
    s, _ = H.SolverFactory.make("FGMRES", "NONE", M,
                               H.SolverParams(tol=1e-30, max_iter=m, restart_size=m))
    x, st = np.zeros(n), H.SolverStats()
    s.solve(M, b, x, st)
    assert st.iterations == m
    assert np.linalg.norm(x - want) <= 1e-11 * np.linalg.norm(want)
