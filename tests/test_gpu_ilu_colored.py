"""ILU(0) on coloured and randomly ordered grids: a few levels of most of the rows, swept by the
whole grid, bit for bit against the oracle, in place too (-m gpu)."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H
from hsps_b200 import problems as P

pytestmark = pytest.mark.gpu


def reordered(side, key):
    """5-point operator on a side x side grid with its rows sorted by `key` (stable)."""
    rp, ci, v = P.varkappa_poisson_2d(side, 1.0, 1)
    n = side * side
    p = np.empty(n, np.int64)
    p[np.argsort(key, kind="stable")] = np.arange(n)
    r, c = p[np.repeat(np.arange(n), np.diff(rp))], p[ci]
    o = np.lexsort((c, r))
    out = np.zeros(n + 1, np.int64)
    out[1:] = np.bincount(r, minlength=n)
    return np.cumsum(out).astype(np.int32), c[o].astype(np.int32), v[o]


def keys(side):
    i, j = np.divmod(np.arange(side * side), side)
    return {"red_black": (i + j) % 2, "four": 2 * (i % 2) + j % 2, "nine": 3 * (i % 3) + j % 3,
            "random": np.random.default_rng(1).permutation(side * side)}


@pytest.mark.parametrize("side,name", [(128, "red_black"), (201, "red_black"), (160, "four"), (301, "nine"),
                                       (257, "random"), (64, "random")])
def test_bitwise(orc, side, name):
    need_gpu()
    import torch

    A = reordered(side, keys(side)[name])
    n = side * side
    M = H.SparseMatrix(n, n, *A)
    I = H.ILUPreconditioner()
    I.setup(M)
    for which in (0, 1):
        nd, ld = I.level_sets(which)
        no, lo = orc.levels(A[0], A[1], which)
        assert nd == no and np.array_equal(ld, lo)
    rc, lu = orc.ilu0(*A)
    assert rc == 0 and np.array_equal(I.factors(), lu)
    r = P.rhs(n, 31, -1.0, 1.0)
    rc, z = orc.ilu_apply(A[0], A[1], lu, r)
    assert np.array_equal(I.apply(r), z)
    t = torch.from_numpy(r).cuda()
    torch.cuda.synchronize()
    I.apply(t, t)
    assert np.array_equal(t.cpu().numpy(), z)
