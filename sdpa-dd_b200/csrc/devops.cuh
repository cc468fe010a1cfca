// Device helpers shared by the Newton-step kernels.
#pragma once
#include "common.cuh"

namespace sddd {

// A . D for a sparse block matrix given as COO (upper-triangle entries in
// input order): Lal::getInnerProduct(SparseMatrix, DenseMatrix),
// sdpa_linear.cpp:202-298 - the first nnz % 4 terms one at a time, then
// groups of four summed with operator+ before one operator+=.
__device__ __forceinline__ dd_t sparse_dot_term(int n, const int *row, const int *col, const dd_t *val, const dd_t *D, int q) {
    const int i = row[q], j = col[q];
    const dd_t v = ld_dd(val + q);
    if (i == j) return dd_mul(v, ld_dd(D + i + (long)n * j));
    return dd_mul(v, dd_add(ld_dd(D + i + (long)n * j), ld_dd(D + j + (long)n * i)));
}
// Number of "+=" steps of that sum, and the e-th step's addend.
__device__ __forceinline__ int sparse_dot_steps(int nnz) { return nnz % 4 + nnz / 4; }
__device__ __forceinline__ dd_t sparse_dot_step(int n, int nnz, const int *row, const int *col, const dd_t *val, const dd_t *D, int e) {
    const int amari = nnz % 4;
    if (e < amari) return sparse_dot_term(n, row, col, val, D, e);
    const int q = amari + 4 * (e - amari);
    dd_t r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = sparse_dot_term(n, row, col, val, D, q + u);
    return dd_add(dd_add(dd_add(r[0], r[1]), r[2]), r[3]);
}
__device__ __forceinline__ dd_t sparse_dot_dense(int n, int nnz, const int *row, const int *col, const dd_t *val, const dd_t *D) {
    dd_t ret = dd_zero();
    const int steps = sparse_dot_steps(nnz);
    for (int e = 0; e < steps; ++e) ret = dd_acc(ret, sparse_dot_step(n, nnz, row, col, val, D, e));
    return ret;
}

// Rdot with one OpenMP thread: templ += x[k] y[k]; return 0 + templ
// (mplapack/Rdot_omp.cpp).  The loads of eight steps go out ahead of
// their terms; the sum's order is unchanged.
__device__ __forceinline__ dd_t seq_dot(long n, const dd_t *x, const dd_t *y) {
    dd_t t = dd_zero();
    long k = 0;
    for (; k + 8 <= n; k += 8) {
        dd_t a[8], b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            a[u] = ld_dd(x + k + u);
            b[u] = ld_dd(y + k + u);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) t = dd_acc(t, dd_mul(a[u], b[u]));
    }
    for (; k < n; ++k) t = dd_acc(t, dd_mul(ld_dd(x + k), ld_dd(y + k)));
    return dd_acc(dd_zero(), t);
}

// Sum of `count` terms in order from zero with "+=" (the reference's
// sequential reductions) by one CTA: all threads form terms into shared
// memory, lane 0 of warp 0 adds them up while the other warps form the next
// chunk.  Only the additions stay a chain (8 dependent FP64 operations a
// term, about 33 ns); loads, gathers and products leave it.  The value is
// returned on thread 0.  Bound by that chain: a 100-term dot takes 5.7 us
// where one thread that also loaded and multiplied took 12.8, the 580-entry C of a
// 100-vertex max-cut 10.5 instead of 198.
constexpr int CHAIN_CHUNK = 512;
constexpr int CHAIN_THREADS = 256;
template <class Term> __device__ __forceinline__ dd_t cta_chain(long count, Term &&term, double2 (*buf)[CHAIN_CHUNK]) {
    const int tid = threadIdx.x;
    auto make = [&](long base, int first, int step, double2 *to) {
        const int len = (int)(count - base < CHAIN_CHUNK ? count - base : CHAIN_CHUNK);
        for (int e = first; e < len; e += step) {
            const dd_t v = term(base + e);
            to[e] = make_double2(v.hi, v.lo);
        }
    };
    make(0, tid, CHAIN_THREADS, buf[0]);
    __syncthreads();
    dd_t t = dd_zero();
    int half = 0;
    for (long base = 0; base < count; base += CHAIN_CHUNK, half ^= 1) {
        if (tid >= 32) {
            make(base + CHAIN_CHUNK, tid - 32, CHAIN_THREADS - 32, buf[half ^ 1]);
        } else if (tid == 0) {
            const int len = (int)(count - base < CHAIN_CHUNK ? count - base : CHAIN_CHUNK);
            const double2 *p = buf[half];
            int e = 0;
            for (; e + 8 <= len; e += 8) {
                double2 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = p[e + u];
#pragma unroll
                for (int u = 0; u < 8; ++u) t = dd_acc(t, dd_make(v[u].x, v[u].y));
            }
            for (; e < len; ++e) t = dd_acc(t, dd_make(p[e].x, p[e].y));
        }
        __syncthreads();
    }
    return t;
}

} // namespace sddd
