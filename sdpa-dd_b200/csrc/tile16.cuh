// A 16 x 16 tile of sequential dd products sum_k a(i,k) b(k,j), one CTA of
// 128 threads, for products too small to give every SM warps enough to hide
// the additions' chains (blas.cu, schur.cu, batched.cu).
//
// Thread (tx, ty) holds entries (ty, tx) and (ty + 8, tx).  An entry's sum is
// a chain (8 dependent FP64 operations a term), so what counts is that
// nothing else lands in it: the loop over k is rolled and carries the
// products of its next step and the operands of the one after in registers
// (in an unrolled loop the compiler places each product directly before its
// addition: 234 cycles a term against 145 here, both chains of a thread), and the next 16 steps'
// operands come from global memory while the current ones are summed.
#pragma once
#include "common.cuh"

namespace sddd {

constexpr int T16 = 16, T16_K = 16, T16_THREADS = 128, T16_CTAS = 7;
constexpr long T16_PIPE_TILES = 2 * 148; // at most this many tiles: the pipelined loop

// Shared memory of one tile: 16 steps of both operands.
struct Tile16 {
    double2 a[T16_K][T16 + 1], b[T16_K][T16 + 1];
};

// la(i, k), lb(j, k): operand entries of the tile's row i / column j, k < K
// (and zero where the tile sticks out of the matrix).  ACONT / BCONT: k is
// the contiguous direction of the operand.  sub: acc - a b, else acc + a b.
// Every product is b * a (operator* commutes bit for bit).
// PIPE: few warps an SM (the form above); otherwise the loop is unrolled and
// the other warps hide the chains, without the moves that carry the products.
template <bool ACONT, bool BCONT, bool SUB, bool PIPE, class LA, class LB>
__device__ __forceinline__ void tile16_sum(Tile16 &S, long K, LA &&la, LB &&lb, dd_t (&acc)[2]) {
    constexpr int PER = T16 * T16_K / T16_THREADS; // operand entries a thread brings
    const int tid = threadIdx.x, tx = tid % T16, ty = tid / T16;
    double2 ra[PER], rb[PER];
    auto fetch = [&](long k0) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + u * T16_THREADS;
            const int ia = ACONT ? e / T16_K : e % T16, ka = ACONT ? e % T16_K : e / T16;
            const int jb = BCONT ? e / T16_K : e % T16, kb = BCONT ? e % T16_K : e / T16;
            ra[u] = k0 + ka < K ? la(ia, k0 + ka) : make_double2(0.0, 0.0);
            rb[u] = k0 + kb < K ? lb(jb, k0 + kb) : make_double2(0.0, 0.0);
        }
    };
    fetch(0);
    for (long k0 = 0; k0 < K; k0 += T16_K) {
        __syncthreads(); // the steps before are summed
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + u * T16_THREADS;
            S.a[ACONT ? e % T16_K : e / T16][ACONT ? e / T16_K : e % T16] = ra[u];
            S.b[BCONT ? e % T16_K : e / T16][BCONT ? e / T16_K : e % T16] = rb[u];
        }
        __syncthreads();
        if (k0 + T16_K < K) fetch(k0 + T16_K);
        const int len = (int)(K - k0 < T16_K ? K - k0 : T16_K);
        if constexpr (!PIPE) {
            auto step = [&](int k) {
                const double2 x = S.b[k][tx], y0 = S.a[k][ty], y1 = S.a[k][ty + 8];
                const dd_t p0 = dd_mul(dd_make(x.x, x.y), dd_make(y0.x, y0.y)), p1 = dd_mul(dd_make(x.x, x.y), dd_make(y1.x, y1.y));
                acc[0] = SUB ? dd_sub(acc[0], p0) : dd_acc(acc[0], p0);
                acc[1] = SUB ? dd_sub(acc[1], p1) : dd_acc(acc[1], p1);
            };
            if (len == T16_K) {
#pragma unroll
                for (int k = 0; k < T16_K; ++k) step(k);
            } else {
                for (int k = 0; k < len; ++k) step(k);
            }
            continue;
        }
        double2 x = S.b[0][tx], y0 = S.a[0][ty], y1 = S.a[0][ty + 8];
        dd_t p0 = dd_mul(dd_make(x.x, x.y), dd_make(y0.x, y0.y)), p1 = dd_mul(dd_make(x.x, x.y), dd_make(y1.x, y1.y));
        x = S.b[1][tx], y0 = S.a[1][ty], y1 = S.a[1][ty + 8];
#pragma unroll 1
        for (int k = 0; k < len; ++k) {
            const int next = min(k + 2, T16_K - 1); // (products past len are not added)
            const dd_t q0 = dd_mul(dd_make(x.x, x.y), dd_make(y0.x, y0.y)), q1 = dd_mul(dd_make(x.x, x.y), dd_make(y1.x, y1.y));
            x = S.b[next][tx], y0 = S.a[next][ty], y1 = S.a[next][ty + 8];
            acc[0] = SUB ? dd_sub(acc[0], p0) : dd_acc(acc[0], p0);
            acc[1] = SUB ? dd_sub(acc[1], p1) : dd_acc(acc[1], p1);
            p0 = q0;
            p1 = q1;
        }
    }
}

} // namespace sddd
