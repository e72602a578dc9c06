"""Division by a stored reciprocal (csrc/exact_div.hpp) against the division, bit for bit: on the
CPU in both types, over random mantissas, mantissas near 1 and 2, and exponents at and around
each limit of its fast path, with zeros, subnormals, infinities and NaN; and FP64 through an
ILU(0) apply on the GPU."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hybrid-sparse-pde-solver_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include <random>
#include <vector>
#include "exact_div.hpp"
using namespace hamlss;

template <typename T, typename B>
B bits(T x) { B b; std::memcpy(&b, &x, sizeof(T)); return b; }

template <typename T, typename B>
long long check(const std::vector<int>& se, const std::vector<int>& de, int mantissa_bits, int rounds, long long& fast) {
    std::mt19937_64 g(7);
    long long bad = 0;
    auto mantissa = [&](int kind) -> T {             // in [1, 2)
        const B m = ((B)1 << mantissa_bits) - 1;
        B f = (B)g() & m;
        if (kind == 1) f &= (B)7;                    // just above 1
        if (kind == 2) f |= m ^ (B)7;                // just below 2
        if (kind == 3) f = 0;
        return (T)1 + (T)std::ldexp((double)f, -mantissa_bits);
    };
    auto one = [&](T s, T d) {
        const T r = recip_of<T>(d), q = div_by<T>(s, d, r), want = s / d;
        fast += DivRange<T>::safe(s) && r != (T)0;
        if (want != want ? q == q : bits<T, B>(q) != bits<T, B>(want)) ++bad;
    };
    for (int round = 0; round < rounds; ++round)
        for (int a : se)
            for (int b : de) {
                const T s = (T)std::ldexp((double)mantissa(round & 3), a) * (g() & 1 ? 1 : -1);
                const T d = (T)std::ldexp((double)mantissa(round >> 2 & 3), b) * (g() & 1 ? 1 : -1);
                one(s, d);
            }
    const T inf = std::numeric_limits<T>::infinity(), nan = std::numeric_limits<T>::quiet_NaN();
    const T odd[] = {(T)0, -(T)0, inf, -inf, nan, std::numeric_limits<T>::denorm_min(), std::numeric_limits<T>::min(),
                     std::numeric_limits<T>::max(), (T)1, (T)-3};
    for (T s : odd)
        for (T d : odd) one(s, d);
    return bad;
}

int main() {
    std::vector<int> s64, d64, s32, d32;
    for (int e : {-1074, -1023, -1022, -800, -624, -623, -622, -300, -53, -1, 0, 1, 52, 300, 575, 576, 577, 578, 1000, 1023}) s64.push_back(e);
    for (int e : {-1074, -1022, -400, -201, -200, -199, -60, -1, 0, 1, 60, 199, 200, 201, 400, 1023}) d64.push_back(e);
    for (int e = -149; e <= 127; e += 3) s32.push_back(e);
    for (int e : {-59, -58, -57, -56, 51, 52, 53, 54}) s32.push_back(e);
    for (int e : {-149, -126, -32, -31, -30, -29, -10, -1, 0, 1, 10, 29, 30, 31, 32, 100, 127}) d32.push_back(e);
    long long fast = 0;
    const long long a = check<double, uint64_t>(s64, d64, 52, 16000, fast);
    const long long fast64 = fast;
    const long long b = check<float, uint32_t>(s32, d32, 23, 4000, fast);
    std::printf("%lld %lld %lld %lld\n", a, b, fast64, fast - fast64);
}
"""


def test_bit_for_bit_on_the_cpu(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    bad64, bad32, fast64, fast32 = map(int, subprocess.run([str(exe)], capture_output=True, text=True,
                                                           check=True).stdout.split())
    assert bad64 == 0 and bad32 == 0
    assert fast64 > 1_000_000 and fast32 > 1_000_000          # the fast path is what was compared


@pytest.mark.gpu
def test_bit_for_bit_through_an_apply():
    # a diagonal matrix: z = r / d (rows of one level, the ring kernel); |d| >= 2^-52, below which
    # the backward sweep refuses a diagonal
    from gpu_util import need_gpu

    need_gpu()
    import hsps_b200 as H

    rng = np.random.default_rng(3)
    n = 4096
    for k in range(12):
        de = rng.choice([-51, -50, -1, 0, 1, 60, 199, 200, 201, 400, 1000], n)
        se = rng.choice([-1074, -1022, -800, -624, -623, -622, -60, 0, 1, 60, 575, 576, 577, 578, 900, 1023], n)
        d = np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), de)
        s = np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), se)
        s[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, np.finfo(float).max]
        d[8:10] = [np.inf, -np.inf]
        I = H.ILUPreconditioner()
        I.setup(H.SparseMatrix(n, n, np.arange(n + 1), np.arange(n), d))
        z = I.apply(s)
        with np.errstate(all="ignore"):
            want = s / d
        ok = (z.view(np.int64) == want.view(np.int64)) | (np.isnan(z) & np.isnan(want))
        assert ok.all(), (s[~ok][:4], d[~ok][:4])
