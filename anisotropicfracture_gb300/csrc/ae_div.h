// An FP64 quotient from a reciprocal at hand (device code; the same operations on the host, for the test).
#pragma once
#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define AE_HD __host__ __device__ __forceinline__
#else
#define AE_HD inline
#endif

namespace ae {

// exponent field of v
AE_HD unsigned exponent_bits(double v) {
#ifdef __CUDA_ARCH__
    return ((unsigned)__double2hiint(v) >> 20) & 0x7ff;
#else
    unsigned long long b;
    std::memcpy(&b, &v, sizeof b);
    return (unsigned)(b >> 52) & 0x7ff;
#endif
}
AE_HD bool zero_bits(double v) {
#ifdef __CUDA_ARCH__
    return (__double_as_longlong(v) << 1) == 0;
#else
    return v == 0.0;
#endif
}

// a / d from inv, which is 1 / d to within four units of 2^-53: the product a inv and one correction by its
// remainder, both fused (Markstein's method: P. W. Markstein, Computation of elementary functions on the IBM
// RISC System/6000 processor, IBM J. Res. Dev. 34 (1990) 111-119).
//
// With u = 2^-53 the product is off by e <= 5 u, so the remainder a - d q is a few units in the last place of
// d q and exact but for a rounding of e u, and the corrected sum is a / d (1 + t), |t| < 32 u^2, before its one
// rounding: the rounded quotient, unless a / d is that near to the middle of two numbers (|t| is less than
// 2^-47 units in the last place).  That holds while nothing under- or overflows; where d, a or the result is
// within 2^64 of the ends of the exponent range, infinite or not a number, it divides.  a = 0 gives a zero,
// whose sign is not kept.
AE_HD double div_by(double a, double d, double inv) {
    const double q = a * inv;
    const double c = fma(fma(-d, q, a), inv, q);
    const unsigned e = exponent_bits(c), ed = exponent_bits(d), ea = exponent_bits(a);
    return ed - 64u < 0x780u && (zero_bits(a) || (e - 64u < 0x780u && ea - 64u < 0x780u)) ? c : a / d;
}

}  // namespace ae
