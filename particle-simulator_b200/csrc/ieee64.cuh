// ieee64.cuh -- square root, reciprocal and quotient rounded to nearest in FP64, without branches.
#pragma once

#include "common.cuh"

namespace dem {

// sqrt, 1 / b and a / b rounded to nearest, for operands whose results and residuals neither
// overflow nor lose bits below 2^-1022 (the callers check ranges and send anything else to the
// operators).  The operators test for such operands each time; without their branches several
// pairs are in flight per thread, and quotients by one divisor share its reciprocal.
//
// tests/test_gpu_ieee64.py compares them with the operators on random operands, on mantissas near 1
// and near 2, and on the square roots and quotients nearest to the midpoints of two doubles.  The square root's error
// before its last rounding is below 2^-102.8 of the result's unit, so only an x whose root lies within
// 37 x 2^-108 of a midpoint could round wrongly; those x = m^2 + k 2^-106 (m odd in units of 2^-53, k = 7 mod 8) are
// enumerated there for |k| <= 513.
//
// The quotient (ulp: of a / b; mantissas in [1, 2)).  q = RN(a RN(1 / b)) is up to 1.5 ulp off, where Markstein's
// theorem asks for 1.  With E = |q - a / b|, the last step's argument is off by at most E m_b / 2 2^-53 for RN(1 / b)
// and, if E > 2 / m_b, when the residual takes 54 bits, 2^-52 / m_b for its rounding: below 2.5 x 2^-53 in all, so
// that only an a / b within that of a midpoint could round wrongly.  There E is 1/2 or 3/2 (to 2.5 x 2^-53).
//   E = 1/2: the residual is exact and the argument off by less than m_b / 4 2^-53 (1 + 2^-50), while a / b is at
//     least 2^-53 / m_b from any midpoint: too near only if m_b >= 2.
//   E = 3/2: a RN(1 / b) is 1 ulp - 2.5 x 2^-53 or more from a / b, so that m_a > 2 - 3 x 2^-52 and 1 / b lies
//     within 0.75 x 2^-53 of its unit of a midpoint.  Such a b has an integer mantissa B < 2^53 that divides
//     2^106 - 1 or 2^106 + 1: 2^53 - 1 (all ones, left to the operators) and 2^53 - 2^27 + 1, which the test takes
//     with the mantissas of a in question.
// Seeds: 2^-20 relative.
__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double rcp_seed(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// v 2^k by the exponent field (v and v 2^k normal): an integer add, off the FP64 pipe.
__device__ __forceinline__ double times_pow2(double v, int k) {
    return __hiloint2double(__double2hiint(v) + (k << 20), __double2loint(v));
}

// RN(sqrt(x)) and h ~ 1 / (2 sqrt(x)): Goldschmidt's coupled iteration (g -> sqrt(x), h -> 1 / (2 sqrt(x)),
// residual r = 1/2 - g h) with the series 1 + r + 3/2 r^2 of (1 - 2 r)^(-1/2) in one step, then one
// correction of g by its exact residual x - g^2 (Markstein 1990).
__device__ __forceinline__ double sqrt_rn(double x, double &h) {
    const double y = rsqrt_seed(x);
    double g = x * y;
    h = times_pow2(y, -1);
    const double r = __fma_rn(-g, h, 0.5);
    const double t = __fma_rn(1.5 * r, r, r);
    g = __fma_rn(g, t, g);
    h = __fma_rn(h, t, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// RN(1 / b) from y within one ulp of it (Markstein 1990), unless every mantissa bit of b is 1.
__device__ __forceinline__ double rcp_last(double b, double y) { return __fma_rn(__fma_rn(-b, y, 1.0), y, y); }

// RN(1 / b): Newton's residual e = 1 - b y and y (1 + e + e^2), then the last step.
__device__ __forceinline__ double rcp_rn(double b) {
    const double y = rcp_seed(b);
    const double e = __fma_rn(-b, y, 1.0);
    return rcp_last(b, __fma_rn(__fma_rn(e, e, e), y, y));
}

// RN(a / b) from y = RN(1 / b): a y corrected by its residual (Markstein 1990; above).
__device__ __forceinline__ double quotient_rn(double a, double b, double y) {
    const double q = a * y;
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

__device__ __forceinline__ bool hi_in(double v, unsigned lo, unsigned hi) {  // exponent range of a positive double
    return (unsigned)__double2hiint(v) - lo < hi - lo;
}
__device__ __forceinline__ bool low_word_ones(double v) { return __double2loint(v) == -1; }
constexpr DEM_HD unsigned hi_of_pow2(int e) { return (unsigned)(e + 1023) << 20; }
// Minimum image, as mic64 (direct_droplet_force_calculator.py:234-240): the subtraction predicated, not selected.
__device__ __forceinline__ void image1(double &d, double L, double halfL) {
    asm("{\n\t.reg .pred p;\n\tsetp.gt.f64 p, %1, %2;\n\t@p sub.rn.f64 %0, %0, %3;\n\t}"
        : "+d"(d)
        : "d"(fabs(d)), "d"(halfL), "d"(copysign(L, d)));
}

}  // namespace dem
