// The dd quotient of dd.h with the same bits on a shorter dependent chain, for
// the diagonal steps of the triangular solves.
//
// dd_div rounds both its double quotients correctly, so any correctly rounded
// quotient gives the same bits.  Here they come from Markstein's correction
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990): with y = RN(1/b) and q
// within one ulp of a/b, fma(fma(-b, q, a), y, q) is a/b correctly rounded.
// The difference of a and its approximation q b is exact (Sterbenz), so
// dd_div's TwoDiff of them needs one subtraction.  All this needs exponents
// away from the ends of the range: outside 2^-400 .. 2^400 (and for a b whose
// significand is all ones) the plain division runs.
// On a B200 a divide is a chain of 127 cycles, a dependent FMA 8; dd_div 299,
// this form with the reciprocal at hand 177.
#pragma once
#include "common.cuh"

namespace sddd {

__device__ __forceinline__ bool mid_range(double a) {
    return (((unsigned)__double2hiint(a) >> 20) & 0x7ffu) - (1023u - 400u) <= 800u;
}
// Significand of all ones (the corrections' one exception).
__device__ __forceinline__ bool all_ones(double b) { return (__double2hiint(b) & 0xfffff) == 0xfffff && __double2loint(b) == -1; }
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
} // namespace sddd
