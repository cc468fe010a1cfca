// Smallest eigenpair of a small symmetric tridiagonal matrix in dd, by one
// warp or one CTA (device code of eig.cu).
#pragma once

#include "common.cuh"

namespace sddd {

// Shared memory of one tri_min_eigenpair of order <= K by NW warps: T scaled
// by a power of two (diagonal, off-diagonal, its reciprocal and square), the
// two-sided recurrences' coefficients and vectors, and the warps' ballots.
template <int K, int NW> struct alignas(16) TriWork {
    dd_t ds[K], es[K], is[K], e2s[K], z[K];
    dd_t ca[2][K], cc[2][K]; // [direction][step's row]: (l - d_i)/e_next and e_prev/e_next
    double2 m[K];            // {d_i, e_{i-1}^2} in double
    double yf[K], yb[K];
    int piv[K];
    unsigned ball[2 * NW];
    dd_t lam, last, nrm2;
    int ok;
};

// Number of eigenvalues of tridiagonal (d, e2 = e^2) below x.
__device__ inline int sturm_count(int k, const dd_t *d, const dd_t *e2, dd_t x) {
    int c = 0;
    dd_t q = dd_sub(d[0], x);
    if (q.hi < 0.0) c++;
    for (int i = 1; i < k; ++i) {
        if (dd_is_zero(q)) q = dd_make(1e-300, 0.0);
        q = dd_sub(dd_sub(d[i], x), dd_div(e2[i - 1], q));
        if (q.hi < 0.0) c++;
    }
    return c;
}

// Whether T has an eigenvalue below x: some leading minor p_i(x) of T - x I
// is negative.  p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1}: one dependent
// FMA a step and no division.  |d|, |x| <= about 1, so the minors grow at
// most as 2^i; a pair that has become tiny is scaled up together every eight
// steps.  m[i] = {d_i, e_{i-1}^2}, m[0].y = 0.
__device__ inline bool tri_below_d(int k, const double2 *m, double x) {
    double p0 = 0.0, p1 = 1.0;
    int sign = 0;
    for (int i = 0; i < k; i += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (i + u < k) {
                const double2 t = m[i + u];
                const double p2 = __fma_rn(t.x - x, p1, -(t.y * p0));
                p0 = p1;
                p1 = p2;
                sign |= __double2hiint(p1);
            }
        }
        if (fabs(p1) < 0x1p-300) {
            p0 *= 0x1p300;
            p1 *= 0x1p300;
        }
    }
    return sign < 0;
}

// a x + b y for dd operands, rounded about once from twice the precision:
// the chain from x to the result is 9 dependent operations, a dd product and
// a dd sum take 17.
__device__ __forceinline__ dd_t dd_dot2(dd_t a, dd_t x, dd_t b, dd_t y) {
    const double p = __dmul_rn(a.hi, x.hi), q = __dmul_rn(b.hi, y.hi);
    const double pe = __fma_rn(a.lo, x.hi, __fma_rn(a.hi, x.lo, __fma_rn(a.hi, x.hi, -p)));
    const double qe = __fma_rn(b.lo, y.hi, __fma_rn(b.hi, y.lo, __fma_rn(b.hi, y.hi, -q)));
    double se, s = ddm::two_sum(p, q, se);
    double e = __dadd_rn(se, __dadd_rn(pe, qe));
    s = ddm::fast_two_sum(s, e, e);
    return dd_make(s, e);
}

// tri_below_d in dd (e2[i] = e_i^2).
__device__ inline bool tri_below_dd(int k, const dd_t *d, const dd_t *e2, dd_t x) {
    dd_t p0 = dd_from(1.0), p1 = dd_sub(d[0], x);
    int sign = __double2hiint(p1.hi);
    for (int i = 1; i < k; ++i) {
        const dd_t p2 = dd_dot2(dd_sub(d[i], x), p1, dd_neg(e2[i - 1]), p0);
        p0 = p1;
        p1 = p2;
        sign |= __double2hiint(p1.hi);
        if ((i & 7) == 0 && fabs(p1.hi) < 0x1p-300) {
            p0 = dd_make(p0.hi * 0x1p300, p0.lo * 0x1p300);
            p1 = dd_make(p1.hi * 0x1p300, p1.lo * 0x1p300);
        }
    }
    return sign < 0;
}

__device__ __forceinline__ dd_t shfl_dd(dd_t v, int src) {
    return dd_make(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
__device__ __forceinline__ dd_t shfl_xor_dd(dd_t v, int m) {
    return dd_make(__shfl_xor_sync(0xffffffffu, v.hi, m), __shfl_xor_sync(0xffffffffu, v.lo, m));
}
// Sum over the warp, the same value in every lane (dd_add commutes bit for
// bit, so both sides of each exchange form the same sum).
__device__ __forceinline__ dd_t warp_sum_dd(dd_t v) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v = dd_add(v, shfl_xor_dd(v, m));
    return v;
}

template <int NW> __device__ __forceinline__ void tri_sync() {
    if (NW == 1)
        __syncwarp();
    else
        __syncthreads();
}

// Index of the first point, over all warps, whose flag is set, or -1.  half
// alternates, so that one barrier a round is enough.
template <int NW> __device__ inline int tri_first_set(bool flag, unsigned *ball, int &half) {
    const unsigned b = __ballot_sync(0xffffffffu, flag);
    if (NW == 1) return __ffs(b) - 1;
    unsigned *hb = ball + half * NW;
    if ((threadIdx.x & 31) == 0) hb[threadIdx.x >> 5] = b;
    tri_sync<NW>();
    half ^= 1;
    const unsigned v = (threadIdx.x & 31) < NW ? hb[threadIdx.x & 31] : 0u;
    const unsigned any = __ballot_sync(0xffffffffu, v != 0u);
    if (any == 0u) return -1;
    const int w = __ffs(any) - 1;
    return 32 * w + __ffs(__shfl_sync(0xffffffffu, v, w)) - 1;
}

// The general path: dd multisection over P = 32 NW points a round, one dd
// Sturm count (k dependent dd divisions) a point, from the double bracket
// [a, b] widened by 2^-40 of the scale when two counts confirm it, else from
// Gershgorin's.
template <int K, int NW> __device__ dd_t tri_multisection(int k, const dd_t *d, const dd_t *e, double a, double b, TriWork<K, NW> &S) {
    const int g = threadIdx.x, P = 32 * NW;
    dd_t *e2 = S.e2s;
    int half = 0;
    dd_t lo = d[0], hi = d[0];
    for (int i = 0; i < k; ++i) {
        dd_t r = dd_zero();
        if (i > 0) r = dd_add(r, dd_abs(e[i - 1]));
        if (i + 1 < k) r = dd_add(r, dd_abs(e[i]));
        lo = dd_min(lo, dd_sub(d[i], r));
        hi = dd_max(hi, dd_add(d[i], r));
    }
    tri_sync<NW>();
    if (g < k - 1) e2[g] = dd_mul(e[g], e[g]);
    tri_sync<NW>();
    dd_t w = dd_sub(hi, lo);
    lo = dd_sub(lo, dd_mul_d(w, 1e-10));
    hi = dd_add(hi, dd_mul_d(w, 1e-10));
    const double PP = (double)(P + 1);
    {
        const double rad = (fabs(lo.hi) + fabs(hi.hi)) * 0x1p-40;
        const dd_t blo = dd_from(a - rad), bhi = dd_from(b + rad);
        bool bad = !(dd_lt(lo, blo) && dd_lt(blo, bhi) && dd_lt(bhi, hi));
        if (!bad && g == 0) bad = sturm_count(k, d, e2, blo) != 0;
        if (!bad && g == 1) bad = sturm_count(k, d, e2, bhi) == 0;
        if (tri_first_set<NW>(bad, S.ball, half) < 0) {
            lo = blo;
            hi = bhi;
        }
    }
    for (int round = 0; round < 40; ++round) {
        const dd_t width = dd_sub(hi, lo);
        // P interior points x_g = lo + width (g+1)/(P+1); the smallest
        // eigenvalue lies below the first x with a non-zero Sturm count,
        // or above x_(P-1) when there is none.
        const dd_t x = dd_add(lo, dd_div_d(dd_mul_d(width, (double)(g + 1)), PP));
        bool below;
        if (!dd_gt(x, lo))
            below = false;
        else if (!dd_lt(x, hi))
            below = true;
        else
            below = sturm_count(k, d, e2, x) >= 1;
        const int first = tri_first_set<NW>(below, S.ball, half);
        dd_t nlo, nhi;
        if (first < 0) {
            nlo = dd_add(lo, dd_div_d(dd_mul_d(width, (double)P), PP));
            nhi = hi;
        } else {
            nhi = dd_add(lo, dd_div_d(dd_mul_d(width, (double)(first + 1)), PP));
            nlo = first == 0 ? lo : dd_add(lo, dd_div_d(dd_mul_d(width, (double)first), PP));
        }
        if (!dd_lt(nlo, nhi) || (dd_eq(nlo, lo) && dd_eq(nhi, hi))) break;
        lo = nlo;
        hi = nhi;
    }
    return dd_mul_d(dd_add(lo, hi), 0.5);
}

// Last component of the unit eigenvector of (d, e) for eigenvalue l: three
// steps of inverse iteration with a partially pivoted tridiagonal solve
// (single thread).  T - l I is factored once; each step solves with the
// factors.
template <int K, int NW> __device__ dd_t tri_last_component(int k, const dd_t *d, const dd_t *e, dd_t l, TriWork<K, NW> &S) {
    dd_t *v = S.z, *dd_ = S.ds, *du = S.es, *du2 = S.is, *dl = S.e2s;
    int *piv = S.piv;
    dd_t tnorm = dd_from(1e-300);
    for (int i = 0; i < k; ++i) tnorm = dd_max(tnorm, dd_abs(d[i]));
    for (int i = 0; i < k; ++i) {
        v[i] = dd_from(1.0);
        dd_[i] = dd_sub(d[i], l);
        du[i] = (i + 1 < k) ? e[i] : dd_zero();
        dl[i] = (i + 1 < k) ? e[i] : dd_zero();
        du2[i] = dd_zero();
    }
    for (int i = 0; i + 1 < k; ++i) {
        if (!dd_lt(dd_abs(dd_[i]), dd_abs(dl[i]))) {
            piv[i] = 0;
            if (dd_is_zero(dd_[i])) dd_[i] = dd_mul_d(tnorm, 1e-32);
            dd_t f = dd_div(dl[i], dd_[i]);
            dl[i] = f;
            dd_[i + 1] = dd_sub(dd_[i + 1], dd_mul(f, du[i]));
        } else {
            piv[i] = 1;
            dd_t f = dd_div(dd_[i], dl[i]);
            dd_[i] = dl[i];
            dl[i] = f;
            dd_t t = du[i];
            du[i] = dd_[i + 1];
            dd_[i + 1] = dd_sub(t, dd_mul(f, dd_[i + 1]));
            if (i + 2 < k) {
                du2[i] = du[i + 1];
                du[i + 1] = dd_neg(dd_mul(f, du[i + 1]));
            }
        }
    }
    if (dd_is_zero(dd_[k - 1])) dd_[k - 1] = dd_mul_d(tnorm, 1e-32);
    for (int it = 0; it < 3; ++it) {
        for (int i = 0; i + 1 < k; ++i) {
            if (piv[i]) {
                dd_t t = v[i];
                v[i] = v[i + 1];
                v[i + 1] = dd_sub(t, dd_mul(dl[i], v[i + 1]));
            } else {
                v[i + 1] = dd_sub(v[i + 1], dd_mul(dl[i], v[i]));
            }
        }
        for (int i = k - 1; i >= 0; --i) {
            dd_t t = v[i];
            if (i + 1 < k) t = dd_sub(t, dd_mul(du[i], v[i + 1]));
            if (i + 2 < k) t = dd_sub(t, dd_mul(du2[i], v[i + 2]));
            v[i] = dd_div(t, dd_[i]);
        }
        dd_t nrm = dd_zero();
        for (int i = 0; i < k; ++i) nrm = dd_acc(nrm, dd_mul(v[i], v[i]));
        nrm = dd_sqrt(nrm);
        for (int i = 0; i < k; ++i) v[i] = dd_div(v[i], nrm);
    }
    return v[k - 1];
}

// The fast path of tri_min_eigenpair; false when the result is not confirmed
// (the double bracket goes to br_a, br_b for the general path).
//   1. multisection in double on the leading minors (tri_below_d);
//   2. the double eigenvector by the two-sided recurrence of (T - l I) z = 0,
//      z_{i+1} = ((l - d_i) z_i - e_{i-1} z_{i-1}) / e_i from both ends to
//      the row r of least residual (a twisted factorisation; the divisions
//      by e_i are taken out into coefficients that all lanes form), and the
//      Rayleigh quotient's correction with the residual in dd: l to about
//      (2^-53)^2;
//   3. the same recurrence in dd to row r and its Rayleigh correction, again
//      until the correction is below 2^-99 of T's scale;
//   4. dd minors at l -+ 2^-92 of the scale: nothing below the one, something
//      below the other.  A second warp checks the l of step 2 beside step 3,
//      and only if that does not do is the final l checked.
// A chain of about 9 us at k = 16 and 12 us at k = 33 on sixteen warps; the
// general path's dd Sturm counts (k dependent dd divisions, eight rounds)
// and three single-thread inverse iterations took 50 to 100 us.
template <int K, int NW>
__device__ bool tri_fast(int k, const dd_t *d, const dd_t *e, const dd_t *ie, TriWork<K, NW> &S, dd_t &lam_out, dd_t &last_out,
                         double &br_a, double &br_b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = threadIdx.x;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = lane; i < k; i += 32) {
        double r = 0.0;
        if (i > 0) r = fabs(e[i - 1].hi);
        if (i + 1 < k) r += fabs(e[i].hi);
        lo = fmin(lo, d[i].hi - r);
        hi = fmax(hi, d[i].hi + r);
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, m));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, m));
    }
    const double big = fmax(fabs(lo), fabs(hi));
    if (!(big > 1e-280 && big < 1e280 && hi > lo)) return false;
    // sc big in [1/2, 1), sc a power of two
    const int ex = ((__double2hiint(big) >> 20) & 0x7ff) - 1022;
    const double sc = __hiloint2double((1023 - ex) << 20, 0), isc = __hiloint2double((1023 + ex) << 20, 0);
    // off-diagonals below 2^-107 of the scale count as zero (one-warp form;
    // Lanczos stops before one arises): bit i set where rows i, i+1 decouple
    unsigned cut = 0u;
    auto tiny = [&](int i) { return NW == 1 && !(fabs(e[i].hi) * sc >= 0x1p-107); };
    if (g < k) {
        const dd_t x = dd_make(d[g].hi * sc, d[g].lo * sc);
        S.ds[g] = x;
        dd_t f = dd_zero(), f2 = f, fi = f, fp = f, fpi = f;
        if (g + 1 < k && !tiny(g)) {
            f = dd_make(e[g].hi * sc, e[g].lo * sc);
            fi = dd_make(ie[g].hi * isc, ie[g].lo * isc);
            f2 = dd_mul(f, f);
        }
        if (g > 0 && !tiny(g - 1)) {
            fp = dd_make(e[g - 1].hi * sc, e[g - 1].lo * sc);
            fpi = dd_make(ie[g - 1].hi * isc, ie[g - 1].lo * isc);
        }
        S.es[g] = f;
        S.e2s[g] = f2;
        S.is[g] = fi;
        S.cc[0][g] = dd_neg(dd_mul(fp, fi));
        S.cc[1][g] = dd_neg(dd_mul(f, fpi));
        S.m[g] = make_double2(x.hi, fp.hi * fp.hi);
    }
    if (NW == 1) cut = __ballot_sync(0xffffffffu, g + 1 < k && tiny(min(g, k - 1)));
    tri_sync<NW>();
    double a = lo * sc, b = hi * sc;
    {
        const double pad = (b - a) * 1e-10;
        a -= pad;
        b += pad;
        constexpr int P = 32 * NW, ROUNDS = NW == 1 ? 11 : 6; // 5 bits a round for one warp, 9 for sixteen
        int half = 0;
        for (int round = 0; round < ROUNDS; ++round) {
            const double step = (b - a) * (1.0 / (P + 1));
            const int first = tri_first_set<NW>(tri_below_d(k, S.m, a + step * (double)(g + 1)), S.ball, half);
            const double na = first == 0 ? a : a + step * (double)(first < 0 ? P : first);
            if (first >= 0) b = a + step * (double)(first + 1);
            a = na;
        }
    }
    br_a = a * isc;
    br_b = b * isc;
    const double l0 = 0.5 * (a + b);
    constexpr double DELTA = 0x1p-92;
    // confirmation of x by the calling warp (lanes 0 and 1)
    auto confirmed = [&](dd_t x) {
        const bool below = tri_below_dd(k, S.ds, S.e2s, dd_add_d(x, (lane & 1) ? DELTA : -DELTA));
        return (__ballot_sync(0xffffffffu, below) & 3u) == 2u;
    };
    dd_t l1 = dd_zero();
    int r = 0, b0 = 0, b1 = k - 1;
    const int dir = lane & 1;
    if (warp < 2) { // both warps alike: one goes on in dd, one confirms
        double *yf = S.yf, *yb = S.yb;
        if (warp == 0) {
            double y = 1.0, yp = 0.0;
            double *Y = dir ? yb : yf;
            if (lane < 2) {
                Y[dir ? k - 1 : 0] = 1.0;
                for (int s = 0; s + 1 < k; ++s) {
                    const int i = dir ? k - 1 - s : s, en = dir ? i - 1 : i;
                    double yn = __fma_rn((l0 - S.ds[i].hi) * S.is[en].hi, y, S.cc[dir][i].hi * yp);
                    if (NW == 1 && (cut >> en & 1u)) yn = 1.0; // the next block starts anew
                    yp = y;
                    y = yn;
                    Y[dir ? i - 1 : i + 1] = yn;
                }
            }
        }
    }
    tri_sync<NW>();
    if (warp < 2) {
        double gbest = INFINITY;
        for (int i = lane; i < k; i += 32) {
            double gm = S.ds[i].hi - l0;
            if (i > 0) gm += S.es[i - 1].hi * S.yf[i - 1] / S.yf[i];
            if (i + 1 < k) gm += S.es[i].hi * S.yb[i + 1] / S.yb[i];
            gm = fabs(gm);
            if (gm < gbest) {
                gbest = gm;
                r = i;
            }
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            const double og = __shfl_xor_sync(0xffffffffu, gbest, m);
            const int orow = __shfl_xor_sync(0xffffffffu, r, m);
            if (og < gbest || (og == gbest && orow < r)) {
                gbest = og;
                r = orow;
            }
        }
        const double fz = 1.0 / S.yf[r], bz = 1.0 / S.yb[r];
        // r's block is rows b0 .. b1
        if (NW == 1 && cut != 0u) {
            b0 = 32 - __clz(cut & ((1u << r) - 1u));
            const unsigned after = cut >> r;
            if (after != 0u) b1 = r + __ffs(after) - 1;
        }
        auto zd = [&](int i) { return i < b0 || i > b1 ? 0.0 : i < r ? S.yf[i] * fz : i == r ? 1.0 : S.yb[i] * bz; };
        double num = 0.0, den = 0.0;
        for (int i = lane; i < k; i += 32) {
            const double z = zd(i);
            dd_t c = dd_mul_d(dd_sub_d(S.ds[i], l0), z);
            if (i > 0) c = dd_add(c, dd_mul_d(S.es[i - 1], zd(i - 1)));
            if (i + 1 < k) c = dd_add(c, dd_mul_d(S.es[i], zd(i + 1)));
            num += z * c.hi;
            den += z * z;
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            num += __shfl_xor_sync(0xffffffffu, num, m);
            den += __shfl_xor_sync(0xffffffffu, den, m);
        }
        l1 = dd_add_dd_exact(l0, num / den);
    }
    if (warp == 0) {
        dd_t l = l1, nrm2 = dd_zero();
        bool done = false;
        for (int it = 0; it < 3 && !done; ++it) {
            for (int i = lane; i < k; i += 32) {
                const dd_t t = dd_sub(l, S.ds[i]);
                S.ca[0][i] = dd_mul(t, S.is[i]);
                if (i > 0) S.ca[1][i] = dd_mul(t, S.is[i - 1]);
            }
            __syncwarp();
            dd_t y = dd_from(1.0), yp = dd_zero();
            const int steps = dir ? b1 - r : r - b0;
            if (lane < 2) {
                int i = dir ? b1 : b0;
                const int inc = dir ? -1 : 1;
                const dd_t *ca = S.ca[dir], *cc = S.cc[dir];
                for (int s = 0; s < steps; ++s, i += inc) {
                    S.z[i] = y;
                    const dd_t yn = dd_dot2(ca[i], y, cc[i], yp);
                    yp = y;
                    y = yn;
                }
                y = dd_div(dd_from(1.0), y);
            }
            __syncwarp();
            const dd_t fi = shfl_dd(y, 0), bi = shfl_dd(y, 1);
            dd_t sq = dd_zero();
            for (int i = lane; i < k; i += 32) {
                const dd_t z = i < b0 || i > b1 ? dd_zero() : i == r ? dd_from(1.0) : dd_mul(S.z[i], i < r ? fi : bi);
                S.z[i] = z;
                sq = dd_add(sq, dd_mul(z, z));
            }
            nrm2 = warp_sum_dd(sq);
            __syncwarp();
            dd_t gm = dd_sub(S.ds[r], l);
            if (r > 0) gm = dd_add(gm, dd_mul(S.es[r - 1], S.z[r - 1]));
            if (r + 1 < k) gm = dd_add(gm, dd_mul(S.es[r], S.z[r + 1]));
            const double dl = gm.hi / nrm2.hi;
            l = dd_add_d(l, dl);
            done = fabs(dl) <= 0x1p-99;
        }
        if (lane == 0) {
            S.lam = l;
            S.last = dd_div(S.z[k - 1], dd_sqrt(nrm2));
            S.ok = done && fabs(dd_sub(l, l1).hi) <= 0.5 * DELTA ? 1 : 0;
            S.piv[0] = done ? 1 : 0;
        }
    }
    if (warp == (NW > 1 ? 1 : 0)) {
        const bool c = confirmed(l1);
        if (lane == 0) S.ball[0] = c ? 1u : 0u;
    }
    tri_sync<NW>();
    const dd_t l = S.lam;
    bool good = S.ok != 0 && S.ball[0] == 1u;
    if (!good) {
        if (S.piv[0] == 0) return false;
        tri_sync<NW>();
        if (warp == 0) {
            const bool c = confirmed(l);
            if (lane == 0) S.ball[0] = c ? 1u : 0u;
        }
        tri_sync<NW>();
        good = S.ball[0] == 1u;
    }
    lam_out = dd_make(l.hi * isc, l.lo * isc);
    last_out = S.last;
    return good;
}

// Smallest eigenvalue of the k x k tridiagonal (d, e), k <= K, and the last
// component of its unit eigenvector (its sign is free), with ie = 1/e; all
// 32 NW threads call, every thread gets the same values, and the arrays are
// shared memory that a barrier has published.
template <int K, int NW>
__device__ void tri_min_eigenpair(int k, const dd_t *d, const dd_t *e, const dd_t *ie, TriWork<K, NW> &S, dd_t &lam, dd_t &last) {
    if (k == 1) {
        lam = d[0];
        last = dd_from(1.0);
        return;
    }
    double a = 0.0, b = 0.0;
    if (tri_fast<K, NW>(k, d, e, ie, S, lam, last, a, b)) return;
    tri_sync<NW>();
    lam = tri_multisection<K, NW>(k, d, e, a, b, S);
    tri_sync<NW>();
    if (threadIdx.x == 0) S.last = tri_last_component<K, NW>(k, d, e, lam, S);
    tri_sync<NW>();
    last = S.last;
    tri_sync<NW>();
}

} // namespace sddd
