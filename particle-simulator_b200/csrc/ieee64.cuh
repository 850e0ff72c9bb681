// ieee64.cuh -- square root, reciprocal and quotient rounded to nearest in FP64, without branches.
#pragma once

#include "common.cuh"

namespace dem {

// sqrt, 1 / b and a / b rounded to nearest, for operands whose results and residuals neither
// overflow nor lose bits below 2^-1022 (the callers check ranges and send anything else to the
// operators).  The operators test for such operands each time; without their branches several
// pairs are in flight per thread, and quotients by one divisor share its reciprocal.
//
// Checked against the operators' results on 2e10 operands (random, and with mantissas near 0 and
// near 1), the quotient also exhaustively in precisions of 5 to 8 bits.  The square root's error before
// its last rounding is below 2^-102.8 of the result's unit, so only an x whose root lies within
// 37 x 2^-108 of a midpoint of two doubles could round wrongly; those x = m^2 + k 2^-106 (m odd in units
// of 2^-53, k = 7 mod 8) were enumerated for |k| <= 513 and agree for every even power of two in range.
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

// RN(a / b) from y = RN(1 / b): a y corrected by its residual (Markstein 1990).
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
