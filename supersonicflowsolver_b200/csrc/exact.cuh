// Division and square root as straight-line code, for kernels whose few warps
// cannot hide the latency of the compiler's own.
//
// A `/` or sqrt() is a sequence with a branch to a slow path, which the compiler
// does not interleave with its neighbours: eight independent FP64 divisions of
// one warp take 8 x 150 cycles on sm_100, eight square roots 8 x 306. The
// functions below have no branch, so independent ones overlap, and several
// numerators share one reciprocal: 110 cycles for a group of FP64 divisions, 80
// for square roots.
//
// FP64 results are the correctly rounded ones, so the bits are those of `/` and
// sqrt():
//  * division (P. Markstein, "Computation of elementary functions on the IBM
//    RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990): with y the
//    reciprocal of b rounded to nearest and q within one ulp of a / b, q + (a -
//    b q) y rounds to the correctly rounded quotient. y comes from the
//    approximate reciprocal by a cubic Newton step and a quadratic one, which
//    rounds it correctly unless b's mantissa is all ones (den_ok excludes it);
//    a y, at most 1.5 ulp off, is corrected twice. A zero numerator keeps its sign
//    over a positive b (the residual is formed negated, b q - a, whose exact zero is
//    +0 and adds nothing to a -0); over a negative one the zero's sign is open.
//  * square root: a cubic step from the approximate reciprocal square root gives
//    a root s within one ulp; the signs of x - s s+ and x - s s- (s+, s- its
//    neighbours; Tuckerman's test, in the same paper) say which of the three is
//    the rounded root.
// Both hold while no operand or intermediate leaves the normal range: the
// caller checks its operands (in_range, zero_or_in_range, den_ok) and takes the
// plain operators otherwise.
//
// FP32: the approximate reciprocal (square root) with one residual correction. The
// quotient's correction is itself good to 2^-22, so it is the rounded one but for
// exact values within 2^-21 ulp of a rounding boundary; the root is within 0.51 ulp
// of the exact value. rn_div corrects the reciprocal too: the rounded quotient, as
// above.
#pragma once
#include <cstdint>

namespace psst {

// 2^-LO <= x < 2^HI, x positive (infinities and NaN are outside)
template <int LO, int HI>
__device__ __forceinline__ bool positive_in_range(double x) {
    return (uint32_t)__double2hiint(x) - ((1023u - LO) << 20) < ((uint32_t)(LO + HI) << 20);
}
template <int LO, int HI>
__device__ __forceinline__ bool positive_in_range(float x) {
    return __float_as_uint(x) - ((127u - LO) << 23) < ((uint32_t)(LO + HI) << 23);
}
// the ranges in which the functions below are used: magnitudes in [2^-400,
// 2^400) (FP64) or [2^-60, 2^60) (FP32), or zero
template <typename R>
__device__ __forceinline__ bool zero_or_in_range(R x) {
    if constexpr (sizeof(R) == 8)
        return positive_in_range<400, 400>(fabs(x)) || x == 0.0;
    else
        return positive_in_range<60, 60>(fabsf(x)) || x == 0.0f;
}
template <typename R>
__device__ __forceinline__ bool den_ok(R b) {
    if constexpr (sizeof(R) == 8)
        // a mantissa of ones only: values an ulp below a round number, such as a
        // temperature settling at 300, have a low word of ones and nothing more (and
        // settled flows are full of them: 25 instead of 20 us an iteration of 120 x 40
        // quads while they took the plain operators)
        return ((uint32_t)__double2loint(b) & ((uint32_t)__double2hiint(b) | 0xfff00000u)) != 0xffffffffu &&
               positive_in_range<400, 400>(fabs(b));
    else
        return positive_in_range<60, 60>(fabsf(b));
}

// 1 / b, correctly rounded
__device__ __forceinline__ double lin_recip(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));  // relative error at most 1e-6
    double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}
__device__ __forceinline__ float lin_recip(float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return y;
}
// a / b given y = lin_recip(b)
__device__ __forceinline__ double lin_quot(double a, double b, double y) {
    double t = a * y;
    t = fma(-fma(b, t, -a), y, t);
    return fma(-fma(b, t, -a), y, t);
}
__device__ __forceinline__ float lin_quot(float a, float b, float y) {
    const float t = a * y;
    return fmaf(-fmaf(b, t, -a), y, t);
}
template <typename R>
__device__ __forceinline__ R lin_div(R a, R b) {
    return lin_quot(a, b, lin_recip(b));
}
// the same with the reciprocal corrected first, which rounds it correctly (of 2 -
// 2^-23 and its like, which the correction could leave at a tie, the approximate
// reciprocal is the rounded one on sm_100): the bits of a / b while 1 / b, a / b and
// the residual b q - a, some 2^-24 of a, are normal numbers, and for a = 0. activate()
// (mlp_net.cuh) has 1 <= b < 2^126 and |a| < 87: b is 2 to all bits where |a| is too
// small for a normal residual, and the halves are exact.
__device__ __forceinline__ float rn_div(float a, float b) {
    float y = lin_recip(b);
    y = fmaf(fmaf(-b, y, 1.0f), y, y);
    return lin_quot(a, b, y);
}
__device__ __forceinline__ double lin_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double s = x * y;
    const double r = fma(-s, 0.5 * y, 0.5);  // s (1 + r + 3/2 r^2) is the root to third order
    s = fma(s, fma(1.5 * r, r, r), s);
    const double up = __longlong_as_double(__double_as_longlong(s) + 1);
    const double dn = __longlong_as_double(__double_as_longlong(s) - 1);
    const double t = fma(-s, up, x) > 0.0 ? up : s;
    return fma(-s, dn, x) <= 0.0 ? dn : t;
}
__device__ __forceinline__ float lin_sqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float s = x * y;
    return fmaf(fmaf(-s, s, x), 0.5f * y, s);
}

}  // namespace psst
