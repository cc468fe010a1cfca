// The dd quotient, square root and reciprocal of dd.h with the same bits on a
// shorter dependent chain, for the pivots of the factorisations and the
// diagonal steps of the triangular solves.
//
// dd_div and dd_sqrt round each of their double quotients correctly, so any
// correctly rounded quotient gives the same bits.  Here they come from
// Markstein's corrections (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): with y within one ulp of 1/b, fma(fma(-b, y, 1), y, y) is 1/b
// correctly rounded unless b's significand is all ones; with y = RN(1/b) and
// q within one ulp of a/b, fma(fma(-b, q, a), y, q) is a/b correctly rounded.
// The difference of a value and its approximation is exact (Sterbenz), so
// dd_div's and dd_sqrt's TwoDiff of such a pair needs one subtraction.  All
// this needs exponents away from the ends of the range: outside 2^-400 ..
// 2^400 (and for a b whose significand is all ones) the plain operations run.
// On a B200 a divide is a chain of 127 cycles, a square root 120, a dependent
// FMA 8; dd_div 299, with the reciprocal at hand 177; dd_sqrt and dd_div(1, .)
// one after the other 606, sqrt_rcp_fast 487.
#pragma once
#include "common.cuh"

namespace sddd {

__device__ __forceinline__ bool mid_range(double a) {
    return (((unsigned)__double2hiint(a) >> 20) & 0x7ffu) - (1023u - 400u) <= 800u;
}
// Significand of all ones (the corrections' one exception).
__device__ __forceinline__ bool all_ones(double b) { return (__double2hiint(b) & 0xfffff) == 0xfffff && __double2loint(b) == -1; }
// RN(1/b) from y0, a few ulps off at most; b in mid_range and not all_ones.
__device__ __forceinline__ double rcp_corrected(double b, double y0) {
    const double y1 = __fma_rn(__fma_rn(-b, y0, 1.0), y0, y0);
    return __fma_rn(__fma_rn(-b, y1, 1.0), y1, y1);
}
// RN(a/b) from y = RN(1/b); a, b in mid_range (or a zero from a sum).
__device__ __forceinline__ double div_corrected(double a, double b, double y) {
    const double q0 = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-b, q0, a), y, q0);
    return __fma_rn(__fma_rn(-b, q1, a), y, q1);
}
// dd_div(a, b) from its first quotient q1 = RN(a.hi / b.hi) and y = RN(1/b.hi):
// r = q1 b is within a factor of two of a, so a.hi - r.hi is exact.
__device__ __forceinline__ dd_t dd_div_rest(dd_t a, dd_t b, double q1, double y) {
    using namespace ddm;
    const dd_t r = dd_mul_d(b, q1);
    const double q2 = div_corrected(add(sub(a.hi, r.hi), add(sub(0.0, r.lo), a.lo)), b.hi, y);
    double e, q = fast_two_sum(q1, q2, e);
    return dd_make(q, e);
}
// l = dd_sqrt(d) and r = dd_div(1, l) in straight line; false where they need
// the plain operations (sqrt_rcp_plain) instead.
__device__ __forceinline__ bool sqrt_rcp_fast(dd_t d, dd_t &l, dd_t &r) {
    using namespace ddm;
    const double a = d.hi, s = __dsqrt_rn(a);
    double y; // 1/sqrt(a) to about 2^-22, then two Newton steps
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
#pragma unroll
    for (int i = 0; i < 2; ++i) y = __fma_rn(__fma_rn(mul(-a, y), y, 1.0), mul(0.5, y), y);
    const double x = rcp_corrected(s, y); // dd_sqrt's 1 / sqrt(a.hi)
    const double ax = mul(a, x);
    double pe, p = two_prod(ax, ax, pe);
    const double t = add(sub(a, p), sub(d.lo, pe)); // high part of d - ax^2
    l = dd_add_dd_exact(ax, mul(t, mul(x, 0.5)));
    const double z = rcp_corrected(l.hi, x);
    r = dd_div_rest(dd_from(1.0), l, z, z);
    return a > 0.0 && mid_range(a) && !all_ones(s) && !all_ones(l.hi);
}
__device__ __forceinline__ void sqrt_rcp_plain(dd_t d, dd_t &l, dd_t &r) {
    l = dd_sqrt(d);
    r = dd_div(dd_from(1.0), l);
}

} // namespace sddd
