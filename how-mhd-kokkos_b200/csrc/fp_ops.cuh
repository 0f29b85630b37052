// fp_ops.cuh -- fused multiply-adds, reciprocals, square roots and quotients of
// the hot kernels, without the branches and the latency of the library's.
#pragma once

#include <cuda_runtime.h>

namespace how {

__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fm(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// FP64 reciprocal, square root and reciprocal square root from the hardware's
// 20-odd-bit approximations (the PTX instructions rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64) and one third-order step of Householder's iteration
// (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation,
// 1970): the residual e of the approximation enters through the series
// 1/(1-e) = 1 + e + e^2 and (1-e)^(-1/2) = 1 + e/2 + 3 e^2/8, whose next term
// is below 2^-59.  The approximations have 21 significant bits (their low words
// are zero), so their squares are exact, and e is rounded once.  Largest errors
// measured: near_recip 0.506 and root_inverse 0.507 units in the last place,
// CUDA's rsqrt 0.507.  recip and root end with the correction by the exact
// remainder (Markstein 1990), which leaves the correctly rounded result.
// The library's sqrt() holds the FP64 pipe for 49 cycles per warp and has a
// latency of 250 cycles (measured on one SM); root's nine operations hold it
// for 18.
//
// Nothing here branches or calls: selects stand in for the ends of the range.

// 1 / x to 0.506 ulp (|x| in [2^-1022, 2^1022)), and correctly rounded
__device__ __forceinline__ double near_recip(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fm(-x, y, 1.0);
    return fm(y, fm(e, e, e), y);
}
__device__ __forceinline__ double recip(double x) {
    const double y = near_recip(x), r = fm(y, fm(-x, y, 1.0), y);
    // 1/x lies next to a midpoint when x's significand is all ones: the result
    // is the value above a power of two, and a tie would leave the power
    const int ones = (__double2hiint(x) & 0xfffff) == 0xfffff && __double2loint(x) == -1;
    return __hiloint2double(__double2hiint(r), __double2loint(r) | ones);
}
__device__ __forceinline__ float near_recip(float x) { return __fdividef(1.0f, x); }

// 1 / sqrt(x) to 0.507 ulp, for finite x >= 2^-1022
__device__ __forceinline__ double root_inverse(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fm(-x, y * y, 1.0);
    return fm(y * e, fm(0.375, e, 0.5), y);
}
__device__ __forceinline__ float root_inverse(float x) { return rsqrtf(x); }

// sqrt(fmax(0, x)), correctly rounded: a NaN gives zero as there; an x below
// 2^-1022 counts as zero
__device__ __forceinline__ double root(double x) {
    const double y = root_inverse(x), g = x * y, r = fm(fm(-g, g, x), 0.5 * y, g);
    const int top = __double2hiint(x);
    const bool end = (unsigned)top - 0x00100000u >= 0x7fe00000u;   // not a normal positive number
    return __hiloint2double(end ? (top == 0x7ff00000 ? top : 0) : __double2hiint(r), end ? 0 : __double2loint(r));
}
__device__ __forceinline__ float root(float x) {
    const float y = rsqrtf(x), g = x * y, r = fm(fm(-g, g, x), 0.5f * y, g);
    return x > 0.0f ? (x < __int_as_float(0x7f800000) ? r : x) : 0.0f;
}

// x / d, correctly rounded, given y = RN(1/d): the steps of div_const
// (how_internal.cuh); a quotient that overflows stays infinite, and one so
// small that its remainder is subnormal is within one unit of 2^-1074 |y|
__device__ __forceinline__ double quot(double x, double d, double y) {
    const double q0 = x * y, q = fm(fm(-q0, d, x), y, q0);
    return (__double2hiint(q0) & 0x7ff00000) == 0x7ff00000 ? q0 : q;
}

// the larger of two non-negative values (doubles order like their bits)
__device__ __forceinline__ double larger(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return __longlong_as_double(x > y ? x : y);
}
__device__ __forceinline__ float larger(float a, float b) { return fmaxf(a, b); }

}  // namespace how
