"""A bounded device-side wait that runs out is reported by the call it happened in (-m gpu).

The kernels that wait (bulk copies, grid barriers) set the context's pinned error word when
a wait runs out, and what they leave behind is not a result.  Here the host sets the word,
as such a kernel would, and no kernel misbehaves.
"""
import ctypes as C

import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import _abi
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


@pytest.fixture
def system():
    """(matrix, its context's word, a right-hand side)"""
    ctx = H.Context.default()
    w = C.POINTER(C.c_int32)()
    assert H.lib().hamlss_ctx_wait_word(ctx.h, C.byref(w)) == 0 and w[0] == 0
    A = H.SparseMatrix(400, 400, *P.poisson_2d(20), ctx=ctx)
    return A, w, P.rhs(400, 1)


@pytest.mark.parametrize("make", [lambda: H.ILUPreconditioner(), lambda: H.JacobiPreconditioner(),
                                  lambda: H.AMGPreconditioner()], ids=["ilu", "jacobi", "amg"])
def test_setup_reports_its_own_wait(system, make):
    A, w, b = system
    M = make()
    w[0] = 1
    with pytest.raises(H.HamlssError) as e:
        M.setup(A)
    assert e.value.code == _abi.ERR_TIMEOUT and w[0] == 0
    assert M.h is None and not M.is_ready()
    A.spmv(b)                                  # the next call is not blamed
    M.setup(A)
    assert np.isfinite(M.apply(b)).all()


def test_failed_setup_leaves_no_word(system):
    A, w, b = system
    v = A.values().copy()
    v[0] = 0.0                                 # a_00: no Jacobi
    A.set_values(v)
    w[0] = 1
    with pytest.raises(H.HamlssError) as e:
        H.JacobiPreconditioner().setup(A)
    assert e.value.code == _abi.ERR_TIMEOUT and w[0] == 0
    with pytest.raises(H.HamlssError) as e:
        H.JacobiPreconditioner().setup(A)
    assert e.value.code == _abi.ERR_ZERO_DIAG


@pytest.mark.parametrize("precond", ["JACOBI", "ILU", "AMG"])
def test_nonfinite_solve_with_a_wait(system, precond):
    # an abandoned kernel's leftovers are often not finite: the wait is what is reported
    A, w, b = system
    s, M = H.SolverFactory.make("FGMRES", precond, A, H.SolverParams(drop_tol=0.0))
    bad = b.copy()
    bad[3] = np.inf
    w[0] = 1
    with pytest.raises(H.HamlssError) as e:
        s.solve(A, bad, np.zeros(400))
    assert e.value.code == _abi.ERR_TIMEOUT and w[0] == 0
    with pytest.raises(H.HamlssError) as e:
        s.solve(A, bad, np.zeros(400))
    assert e.value.code == _abi.ERR_NONFINITE
    A.spmv(b)
    x = np.zeros(400)
    assert s.solve(A, b, x)


@pytest.mark.parametrize("poison", [False, True])
def test_adaptive_with_a_wait(system, poison):
    A, w, b = system
    b = b.copy()
    if poison:
        b[3] = np.inf
    w[0] = 1
    with pytest.raises(H.HamlssError) as e:
        H.AdaptiveSelector(H.SolverParams()).solve(A, b, np.zeros(400))
    assert e.value.code == _abi.ERR_TIMEOUT and w[0] == 0
    A.spmv(np.ones(400))


def test_every_other_call_takes_its_word(system):
    A, w, b = system
    M = H.ILUPreconditioner()
    M.setup(A)
    for call in (lambda: A.spmv(b), lambda: M.apply(b), lambda: H.amg_aggregate(A),
                 lambda: H.AdaptiveSelector().extract_features(A)):
        w[0] = 1
        with pytest.raises(H.HamlssError) as e:
            call()
        assert e.value.code == _abi.ERR_TIMEOUT and w[0] == 0
        call()
