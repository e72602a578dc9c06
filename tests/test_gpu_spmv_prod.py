"""FP64 SpMV of operators with more than 5.5 entries a row (products left in shared memory,
added in column order): bit for bit against the plain loop at the edges of its tiles (512
products a warp, 256 a load, up to 32 rows a warp) and of its row shares (-m gpu)."""
import numpy as np
import pytest

from gpu_util import need_gpu
import hsps_b200 as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    need_gpu()


def from_lengths(lengths, m, seed):
    rng = np.random.default_rng(seed)
    rp = np.zeros(len(lengths) + 1, np.int32)
    rp[1:] = np.cumsum(lengths)
    ci = np.concatenate([np.sort(rng.choice(m, size=k, replace=False)) for k in lengths] or [np.zeros(0, int)])
    v = rng.standard_normal(rp[-1]) * 10.0 ** rng.integers(-8, 9, rp[-1])
    return rp, ci.astype(np.int32), v


def lengths(name, n, rng):
    if name == "uniform":
        return rng.integers(0, 40, n)
    if name == "empty_mostly":
        return np.where(rng.random(n) < 0.1, 90, 0)
    if name == "one_long":
        out = np.full(n, 7)
        out[n // 2] = 900
        return out
    return np.full(n, int(name))


SHAPES = [(1, "6"), (2, "600"), (31, "16"), (32, "16"), (33, "16"), (1000, "uniform"), (2500, "255"),
          (2500, "256"), (2500, "257"), (700, "511"), (700, "512"), (700, "513"), (20000, "6"), (20011, "uniform"),
          (20011, "empty_mostly"), (9000, "one_long"), (40000, "13"), (40001, "uniform"), (599, "17"), (19000, "27")]


@pytest.mark.parametrize("n,name", SHAPES, ids=[f"{n}_{k}" for n, k in SHAPES])
def test_bitwise(n, name):
    rng = np.random.default_rng(n)
    A = from_lengths(lengths(name, n, rng), max(n, 1000), n)
    m = max(n, 1000)
    M = H.SparseMatrix(n, m, *A)
    x = rng.standard_normal(m)
    y = M.spmv(x)
    ref = np.zeros(n)
    for i in range(n):                       # column order, separate multiply and add
        s = np.float64(0.0)
        for k in range(A[0][i], A[0][i + 1]):
            s = s + A[2][k] * x[A[1][k]]
        ref[i] = s
    assert np.array_equal(y, ref)


def test_nonfinite_entries_stay_in_their_rows():
    A = from_lengths(np.full(3000, 12), 3000, 1)
    A[2][5] = np.inf
    A[2][12 * 700 + 3] = np.nan
    x = np.ones(3000)
    y = H.SparseMatrix(3000, 3000, *A).spmv(x)
    bad = ~np.isfinite(y)
    assert np.array_equal(np.flatnonzero(bad), [0, 700])


def grouped(name, rng):
    """Row lengths with neighbouring long rows, at both sides of the rule that leaves them to
    a lane a row."""
    if name == "long_at_the_end":
        return np.concatenate([np.full(20011, 8), np.full(19, 900)])
    if name == "long_in_front":
        return np.concatenate([np.full(50, 900), np.full(20000, 8)])
    if name == "uneven":                     # long, short and empty rows side by side
        out = np.full(20000, 7)
        out[5000:5064] = rng.integers(0, 600, 64)
        out[9000:9032:2] = 997
        out[9001:9033:2] = 0
        return out
    if name == "few":                        # too few to matter
        return np.concatenate([np.full(9000, 9), np.full(6, 900), np.full(9000, 9)])
    return np.concatenate([np.full(3000, 50), np.full(64, 1500), np.full(3000, 50)])   # "wide"


@pytest.mark.parametrize("name", ["long_at_the_end", "long_in_front", "uneven", "few", "wide"])
def test_neighbouring_long_rows_bitwise(name):
    rng = np.random.default_rng(7)
    ln = grouped(name, rng)
    n, m = len(ln), 30000
    A = from_lengths(ln, m, 11)
    x = rng.standard_normal(m)
    y = H.SparseMatrix(n, m, *A).spmv(x)
    ref = np.zeros(n)
    prod = A[2] * x[A[1]]
    for k in range(int(ln.max())):           # column order, every row at once
        has = ln > k
        ref[has] = ref[has] + prod[A[0][:-1][has] + k]
    assert np.array_equal(y, ref)
