"""FGMRES' multi-dots of few vectors at the sizes where a thread an entry takes over (524,288
entries, up to 8 vectors), both sides of each, and below (-m gpu).  The yardstick and its bound
are test_gpu_mdot.py's."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P
from test_gpu_mdot import krylov_minimiser, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(131071, 5), (131072, 1), (131072, 5), (131073, 4), (524287, 8), (524288, 9),
                                 (600001, 8)])
def test_one_cycle(orc, n, m):
    need_gpu()
    csr = matrix(n)
    M = H.SparseMatrix(n, n, *csr)
    b = P.rhs(n, 6, -1.0, 1.0)
    want = krylov_minimiser(lambda x: orc.spmv(*csr, x), b, m)
    s, _ = H.SolverFactory.make("FGMRES", "NONE", M, H.SolverParams(tol=1e-30, max_iter=m, restart_size=m))
    x, st = np.zeros(n), H.SolverStats()
    s.solve(M, b, x, st)
    assert st.iterations == m
    assert np.linalg.norm(x - want) <= 1e-11 * np.linalg.norm(want)
