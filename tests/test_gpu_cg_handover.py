"""The persistent CG iteration across its launches (-m gpu): the state that travels through
memory between them leaves no trace in the results.

A matrix whose blocks hold 256 rows gives the two-launch iteration's bits, trip for trip.  The
same system with stored zeros in the rows of one block no longer fits the block's shared memory
and takes the two-launch iteration; the zeros change no sum.  So both must agree bit for bit
after any number of trips; the launches' names in the profiler show that both forms ran.
"""
import ctypes as C

import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def with_zeros(A, rows, per_row):
    """A with `per_row` stored zeros in each of `rows`, at columns the row does not have."""
    rp, ci, v = A
    n = len(rp) - 1
    r = np.repeat(np.arange(n, dtype=np.int64), np.diff(rp))
    er, ec = [], []
    for i in rows:
        free = np.setdiff1d(np.arange(n), ci[rp[i]:rp[i + 1]])[:per_row]
        er.append(np.full(len(free), i))
        ec.append(free)
    r = np.concatenate([r] + er)
    c = np.concatenate([ci] + ec)
    v = np.concatenate([v, np.zeros(len(r) - len(v))])
    o = np.lexsort((c, r))
    out = np.zeros(n + 1, np.int64)
    out[1:] = np.bincount(r, minlength=n)
    return np.cumsum(out).astype(np.int32), c[o].astype(np.int32), v[o]


def solve(A, precond, b, trips):
    """(x, stats, launches by name) after `trips` trips"""
    n = len(A[0]) - 1
    M = H.SparseMatrix(n, n, *A)
    s, _ = H.SolverFactory.make("CG", precond, M, H.SolverParams(tol=1e-300, max_iter=trips))
    L, ctx = H.lib(), M.ctx
    L.hamlss_profile_enable(ctx.h, 1, 3 * trips + 1000)
    x, st = np.zeros(n), H.SolverStats()
    s.solve(M, b, x, st)
    names, count = np.zeros(64 * 32, np.uint8), np.zeros(64, np.int32)
    ms, by, k = np.zeros(64), np.zeros(64), C.c_int32()
    L.hamlss_profile_read(ctx.h, 64, names.ctypes.data, count.ctypes.data, ms.ctypes.data, by.ctypes.data, C.byref(k))
    L.hamlss_profile_enable(ctx.h, 0, 0)
    launches = {bytes(names[32 * i:32 * i + 32]).split(b"\0")[0].decode(): int(count[i]) for i in range(k.value)}
    return x, st, launches


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
@pytest.mark.parametrize("side,sigma,trips,least", [
    (32, 3.5, 4500, 2),          # one cluster, 4,096 trips a launch
    (64, 3.5, 4500, 2),
    (173, 1.0, 100, 1),          # a block per SM, 1,024 trips a launch
    (173, 2.5, 1024, 1),
    (173, 2.5, 1025, 2),
    (173, 2.5, 2100, 3),
])
def test_same_bits_as_two_launches_a_trip(side, sigma, trips, least, precond):
    A = P.varkappa_poisson_2d(side, sigma, 1)
    n = side * side
    b = P.rhs(n, 2)
    x, st, one = solve(A, precond, b, trips)
    y, su, two = solve(with_zeros(A, range(256), 140), precond, b, trips)
    assert one.get("cg_trips", 0) >= least and "cg_update" not in one, one
    assert "cg_trips" not in two and two.get("cg_update", 0) >= min(trips, 100), two
    assert st.iterations == su.iterations and st.restarts == su.restarts
    assert st.final_residual == su.final_residual
    assert np.array_equal(x, y)
