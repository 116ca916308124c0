// Correctly rounded division by a divisor that many dividends share: its
// reciprocal, correctly rounded, and two fused-multiply-add corrections, which
// end in the correctly rounded quotient (P. W. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34 (1990): with y = RN(1/b), a q within one ulp of a/b and r = a - b q by a
// fused multiply-add, RN(q + r y) = RN(a/b)). 40 cycles of dependent latency
// instead of a division's 113. Operands outside [2^-500, 2^500], where a step
// could leave the normal range, divide.
#pragma once

#include "device_util.cuh"

namespace tns {

// A divisor prepared once for many dividends. Complex (Smith's division, as
// System.Numerics.Complex divides): ratio of the smaller to the larger part
// and the real divisor both quotients share.
struct Divisor {
    double b, y;      // the (real) divisor and its reciprocal
    double ratio;     // complex only
    int re_larger;    // complex only
    int safe;         // the reciprocal form may be used
};

// Exponent in [-500, 500] (no zero, subnormal, infinity or NaN).
__device__ __forceinline__ bool in_range(double v) {
    return ((unsigned)__double2hiint(v) & 0x7ff00000u) - ((1023u - 500u) << 20) <= (1000u << 20);
}
__device__ __forceinline__ Divisor make_divisor(double v) {
    Divisor d;
    d.b = v;
    d.safe = in_range(v);
    d.y = d.safe ? __drcp_rn(v) : 0.0;
    d.ratio = 0.0;
    d.re_larger = 0;
    return d;
}
__device__ __forceinline__ Divisor make_divisor(double2 v) {
    const bool re_larger = fabs(v.y) < fabs(v.x);
    const double big = re_larger ? v.x : v.y, small = re_larger ? v.y : v.x;
    const double ratio = __ddiv_rn(small, big);
    Divisor d = make_divisor(add_rn(big, mul_rn(small, ratio)));
    d.ratio = ratio;
    d.re_larger = re_larger;
    return d;
}
// The quotient for a safe divisor; false when the dividend is out of range.
__device__ __forceinline__ double quotient_fast(double a, const Divisor& d) {
    const double q0 = mul_rn(a, d.y);
    const double q1 = fma(fma(-d.b, q0, a), d.y, q0);
    return fma(fma(-d.b, q1, a), d.y, q1);
}
__device__ __forceinline__ bool divide_fast(double x, const Divisor& d, double& y) {
    y = quotient_fast(x, d);
    return in_range(x);
}
__device__ __forceinline__ double2 numerators(double2 x, const Divisor& d) {
    // (a + ib) / (c + id): |d| < |c|: ((a + b r) / den, (b - a r) / den), r = d / c;
    // else ((b + a r) / den, (-a + b r) / den), r = c / d.
    const double p = d.re_larger ? x.x : x.y, q = d.re_larger ? x.y : x.x;
    const double t = mul_rn(p, d.ratio);
    return make_double2(add_rn(p, mul_rn(q, d.ratio)), add_rn(d.re_larger ? q : -q, d.re_larger ? -t : t));
}
__device__ __forceinline__ bool divide_fast(double2 x, const Divisor& d, double2& y) {
    const double2 nm = numerators(x, d);
    y = make_double2(quotient_fast(nm.x, d), quotient_fast(nm.y, d));
    return in_range(nm.x) & in_range(nm.y);
}
__device__ __forceinline__ double divide(double x, const Divisor& d) { return __ddiv_rn(x, d.b); }
__device__ __forceinline__ double2 divide(double2 x, const Divisor& d) {
    const double2 nm = numerators(x, d);
    return make_double2(__ddiv_rn(nm.x, d.b), __ddiv_rn(nm.y, d.b));
}

}  // namespace tns
