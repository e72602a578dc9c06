"""A request on a solve lane stays within the footprint it was admitted with (-m gpu): the peak
of the device's memory pool while the server solves it.  Patterns whose ILU(0) rows are padded
to their longest one, and an AMG setup whose products take a dense right operand."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import _abi
from hsps_b200 import problems as P
from hsps_b200.serve import Server

pytestmark = pytest.mark.gpu


def csr(n, r, c, v):
    o = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.bincount(r, minlength=n)
    return np.cumsum(rp).astype(np.int32), c[o].astype(np.int32), v[o]


def one_long_row():
    """Unsymmetric grid operator, one row with 14 entries below the diagonal."""
    rp, ci, v = P.varkappa_poisson_2d(250, 1.0, 3)
    n = 62500
    r = np.repeat(np.arange(n), np.diff(rp))
    v = np.where(ci > r, 0.5 * v, v)
    m = n // 2
    return csr(n, np.concatenate([r, np.full(12, m)]), np.concatenate([ci, m - 5000 - 700 * np.arange(12)]),
               np.concatenate([v, np.full(12, -1e-3)]))


def nine_lower():
    n = 60000
    r, c = [np.arange(n)], [np.arange(n)]
    for o in [s * (200 + 3 * j) for j in range(9) for s in (-1, 1)]:
        i = np.arange(max(0, -o), min(n, n - o))
        r.append(i)
        c.append(i + o)
    r, c = np.concatenate(r), np.concatenate(c)
    v = np.where(r == c, 10.0, np.where(c > r, -0.2, -0.4))
    return csr(n, r, c, v)


def weak_diagonal():
    rp, ci, v = P.varkappa_poisson_2d(130, 1.0, 3)
    r = np.repeat(np.arange(130 * 130), np.diff(rp))
    return rp, ci, np.where(ci == r, 0.25 * v, v)


@pytest.mark.parametrize("name,make,state,over", [
    ("one_long_row", one_long_row, 1, {}),
    ("nine_lower", nine_lower, 1, {}),
    ("nine_lower_m5", nine_lower, 1, dict(restart_size=5)),
    ("weak_diagonal", weak_diagonal, 2, dict(max_iter=60)),
], ids=lambda a: a if isinstance(a, str) else "")
def test_peak_within_estimate(name, make, state, over):
    need_gpu()
    rt = pytest.importorskip("cuda.bindings.runtime")
    drv = pytest.importorskip("cuda.bindings.driver")
    attr = rt.cudaMemPoolAttr
    pool = rt.cudaDeviceGetDefaultMemPool(0)[1]
    used = lambda a: int(rt.cudaMemPoolGetAttribute(pool, a)[1])  # noqa: E731
    A = make()
    n = len(A[0]) - 1
    kw = dict(tol=1e-10, max_iter=4000, restart_size=30, drop_tol=0.0, precision=_abi.MIXED, amg_omega=2.0 / 3.0,
              amg_coarse_limit=512, amg_levels=25, amg_stall_ratio=0.75, ladder_mode=3)
    kw.update(over)
    with Server(slots=1, batch_max_rows=0) as srv:
        before = used(attr.cudaMemPoolAttrUsedMemCurrent)
        rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, drv.cuuint64_t(0))
        _, st = srv.submit(*A, P.rhs(n, 1), params=H.SolverParams(**kw)).wait(timeout=100)
        peak = used(attr.cudaMemPoolAttrUsedMemHigh) - before
        estimate = srv.report()["peak_admitted_bytes"]
    assert st.state_used == state            # the rung whose memory is meant
    assert 0 < peak <= estimate, (peak, estimate)
