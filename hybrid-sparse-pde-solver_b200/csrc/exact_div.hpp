// exact_div.hpp -- division by a stored reciprocal, correctly rounded (the triangular sweeps);
// also compiled for the CPU, where a test compares it with the division.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define HAMLSS_HD __host__ __device__ __forceinline__
#else
#define HAMLSS_HD inline
#endif

namespace hamlss {

// s / d given r = 1 / d (rounded; 0 when d is not in [2^-max_exp, 2^max_exp]): Markstein's
// correction (IBM J. Res. Dev. 34, 1990) applied twice.  q0 = s r is within 2 ulp, q1 is a
// faithful quotient, and for a faithful quotient and a correctly rounded reciprocal
// q1 + r (s - d q1), with the remainder exact in an FMA, is the correctly rounded one -- s / d
// bit for bit.  Exponents that could under- or overflow on the way, zeros, infinities and
// NaN take the division.  On the sweep's critical path: 5 dependent operations (~45 cycles)
// for the division's ~115.
template <typename T>
struct DivRange;
template <>
struct DivRange<double> {
    static constexpr int max_exp = 200;
    static HAMLSS_HD bool safe(double s) {
#ifdef __CUDA_ARCH__
        const unsigned hi = (unsigned)__double2hiint(s);
#else
        uint64_t b;
        std::memcpy(&b, &s, 8);
        const unsigned hi = (unsigned)(b >> 32);
#endif
        return (hi >> 20 & 0x7ff) - 400u < 1200u;                               // 2^-623 .. 2^577
    }
};
template <>
struct DivRange<float> {
    static constexpr int max_exp = 30;
    static HAMLSS_HD bool safe(float s) {
#ifdef __CUDA_ARCH__
        const unsigned b = __float_as_uint(s);
#else
        uint32_t b;
        std::memcpy(&b, &s, 4);
#endif
        return (b >> 23 & 0xff) - 70u < 110u;                                   // 2^-57 .. 2^53
    }
};
HAMLSS_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
HAMLSS_HD float fma_rn(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return std::fmaf(a, b, c);
#endif
}

template <typename T>
HAMLSS_HD T recip_of(T d) {
    const T big = (T)ldexp(1.0, DivRange<T>::max_exp), a = d < T(0) ? -d : d;
    return a >= T(1) / big && a <= big ? T(1) / d : T(0);
}

template <typename T>
HAMLSS_HD T div_by(T s, T d, T r) {
    if (DivRange<T>::safe(s) && r != T(0)) {
        const T q0 = s * r;
        const T q1 = fma_rn(fma_rn(-d, q0, s), r, q0);
        return fma_rn(fma_rn(-d, q1, s), r, q1);
    }
    return s / d;
}

}  // namespace hamlss
