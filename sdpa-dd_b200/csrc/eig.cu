// Step-length eigenvalue lambda_min(L D L^T) per SDP block
// (Jal::getMinEigen, sdpa_jordan.cpp:55-88):
//   n > 20   Lanczos of Lal::getMinEigen (sdpa_linear.cpp:27-122): same start
//            vector, recurrences, checkpoint and stopping rules.  The sums of
//            the three matrix-vector products and the two dot products run
//            split over lanes, warps and the CTAs of a cluster (the
//            reference's own sums follow its OpenMP threads); the k x k
//            tridiagonal eigenproblem of a checkpoint is tri_eig.cuh's (the
//            reference uses implicit QR, Rsteqr; both give the eigenvalue
//            and the last eigenvector component to dd rounding).
//   n <= 20  M = L (D L^T) by two Rgemm, then the smallest eigenvalue of the
//            lower triangle of M (the reference's Rsyev "N","L") by
//            Householder tridiagonalisation (one warp) and tri_eig.cuh.
// The whole Lanczos loop runs in one cluster per block: no host round trip
// per step.
#include "newton.h"

#include <algorithm>

#include <cooperative_groups.h>

#include "blas.h"
#include "devops.cuh"
#include "eig_kernels.cuh"
#include "prof.h"
#include "tri_eig.cuh"

namespace sddd {

namespace cg = cooperative_groups;

// QD double-vs-dd comparisons (dd_inline.h operator< / operator>)
__device__ __forceinline__ bool d_lt_dd(double a, dd_t b) { return a < b.hi || (a == b.hi && b.lo > 0.0); }
__device__ __forceinline__ bool d_gt_dd(double a, dd_t b) { return a > b.hi || (a == b.hi && b.lo < 0.0); }

namespace {

constexpr int LZ_WARPS = LZ_THREADS / 32;
constexpr int LZ_CHUNK = 8;     // rows a warp takes together
constexpr int LZ_CLUSTER = 16;  // most CTAs of a cluster

// Compensated dot product of dd operands (Ogita, Rump and Oishi's Dot2 with
// the operands' low parts in the error term): the running sum's chain is one
// addition a term, twelve FP64 operations against dd_acc(dd_mul)'s twenty,
// and the sum is as if rounded once from twice the working precision.
struct DotAcc {
    double s = 0.0, e = 0.0;
    __device__ __forceinline__ void term(double2 a, double2 b) {
        const double p = __dmul_rn(a.x, b.x);
        double pe = __fma_rn(a.x, b.x, -p);
        pe = __fma_rn(a.x, b.y, pe);
        pe = __fma_rn(a.y, b.x, pe);
        double se;
        s = ddm::two_sum(s, p, se);
        e = __dadd_rn(e, __dadd_rn(pe, se));
    }
    __device__ __forceinline__ dd_t value() const {
        double lo, hi = ddm::fast_two_sum(s, e, lo);
        return dd_make(hi, lo);
    }
};

struct alignas(16) LanczosShared {
    dd_t diag[LZ_KMAX], off[LZ_KMAX], ioff[LZ_KMAX];
    TriWork<LZ_KMAX, LZ_WARPS> tri;
    dd_t psum[LZ_WARPS * LZ_CHUNK];
    dd_t pa[LZ_CLUSTER], pr[LZ_CLUSTER];
};

// A vector the products read: in shared memory (every CTA holds all of it),
// or, for orders whose vectors do not fit there, in global memory (read past
// L1, which is not coherent between the CTAs).
template <bool SMEM> __device__ __forceinline__ double2 lz_ld(const dd_t *v, long i) {
    const double2 *p = reinterpret_cast<const double2 *>(v) + i;
    return SMEM ? *p : __ldcg(p);
}
__device__ __forceinline__ double2 mat_ld(const dd_t *p) { return __ldg(reinterpret_cast<const double2 *>(p)); }

// Eight rows i0 .. i0+7 of a product with v, part `part` of 2^lp of the
// terms: lane (row, phase) takes every (4 2^lp)-th term.  FULL: rows of M v;
// LOWER: of M's lower triangle; LOWER_T: of its transpose (row i is column i
// from the diagonal down).  A load instruction covers 128 contiguous bytes of
// each of 4 columns (LOWER_T: 64 bytes of each of 8, the rest of the line at
// the next step).  Every lane of a row returns the part's sum.
enum { LZ_FULL, LZ_LOWER, LZ_LOWER_T };
template <int FORM, bool SMEM> __device__ __forceinline__ dd_t lz_rows(const dd_t *M, int n, int i0, int part, int lp, const dd_t *v) {
    const int lane = threadIdx.x & 31, i = i0 + (lane & 7), step = 4 << lp;
    const int end = i >= n ? 0 : FORM == LZ_LOWER ? i + 1 : n;
    const long sj = FORM == LZ_LOWER_T ? 1 : n; // from one term to the next
    const dd_t *Mi = FORM == LZ_LOWER_T ? M + (long)n * i : M + i;
    DotAcc acc;
    int j = part * 4 + (lane >> 3);
    if (FORM == LZ_LOWER_T) j += i0;
    // the loads of eight terms in flight, then of two
    for (; j + 7 * step < end; j += 8 * step) {
        double2 a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int ju = j + u * step;
            a[u] = FORM == LZ_LOWER_T && ju < i ? make_double2(0.0, 0.0) : mat_ld(Mi + sj * ju);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) acc.term(a[u], lz_ld<SMEM>(v, j + u * step));
    }
    for (; j + step < end; j += 2 * step) {
        const double2 a0 = FORM == LZ_LOWER_T && j < i ? make_double2(0.0, 0.0) : mat_ld(Mi + sj * j);
        const double2 a1 = FORM == LZ_LOWER_T && j + step < i ? make_double2(0.0, 0.0) : mat_ld(Mi + sj * (j + step));
        acc.term(a0, lz_ld<SMEM>(v, j));
        acc.term(a1, lz_ld<SMEM>(v, j + step));
    }
    for (; j < end; j += step)
        if (FORM != LZ_LOWER_T || j >= i) acc.term(mat_ld(Mi + sj * j), lz_ld<SMEM>(v, j));
    dd_t t = acc.value();
    t = dd_add(t, shfl_xor_dd(t, 8));
    return dd_add(t, shfl_xor_dd(t, 16));
}

// The Lanczos loop of one block by one cluster: CTA r of R owns the 8-row
// chunks r, r + R, ... (the triangular products' work then spreads evenly),
// forms those rows of each product and stores them into every CTA's copy of
// the vector; four cluster barriers a step (after w = L^T q, tmp = X w,
// w = L tmp with the parts of q.w, and r with the parts of r.r).  Every CTA
// holds the same scalars, bit for bit (the same operations on the same
// values), so the CTAs agree on every branch without a broadcast.
// Bound by latency up to n of about 200 (barriers, the folds of partial sums
// and the checkpoints' tridiagonal solves, 9 - 12 us each), by the L2 reads
// of one GPC beyond.  One CTA whose threads each ran a row's whole chain of n
// dependent dd sums took 1.20 / 1.98 / 3.73 / 10.6 / 24.1 ms at n = 30 / 100
// / 200 / 500 / 777 (random L D L^T, 16 to 38 steps); this form 0.24 / 0.34 /
// 0.45 / 0.88 / 1.74 ms.
template <bool SMEM>
__global__ void __launch_bounds__(LZ_THREADS) lanczos_kernel(const int *blk_ids, int nb, const int *sizes, const long *off, const dd_t *Lsp,
                                                             const dd_t *Dsp, const dd_t *Lsp2, const dd_t *Dsp2, dd_t *work, long work_stride, dd_t *out) {
    extern __shared__ double2 lz_smem[];
    LanczosShared &S = *reinterpret_cast<LanczosShared *>(lz_smem);
    cg::cluster_group cl = cg::this_cluster();
    const int R = (int)cl.num_blocks(), rank = (int)cl.block_rank(), cid = (int)blockIdx.x / R;
    const bool second = cid >= nb;
    const int b = blk_ids[second ? cid - nb : cid];
    const int n = sizes[b];
    const dd_t *L = (second ? Lsp2 : Lsp) + off[b], *X = (second ? Dsp2 : Dsp) + off[b];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunks = (n + LZ_CHUNK - 1) / LZ_CHUNK;
    const int nch = rank < chunks ? (chunks - rank - 1) / R + 1 : 0, nown = nch * LZ_CHUNK;
    // q, w and tmp (tmp also carries r between the steps), then this CTA's
    // rows of w and of the previous q
    dd_t *local = reinterpret_cast<dd_t *>(&S + 1), *q, *w, *tmp, *wl, *ql;
    if (SMEM) {
        q = local, w = q + n, tmp = w + n, wl = tmp + n, ql = wl + (chunks + R - 1) / R * LZ_CHUNK;
    } else {
        q = work + (long)cid * work_stride, w = q + n, tmp = w + n;
        wl = local, ql = wl + (chunks + R - 1) / R * LZ_CHUNK;
    }
    // global row of own slot s (may be >= n in the last chunk)
    auto row_of = [&](int s) { return (rank + R * (s >> 3)) * LZ_CHUNK + (s & 7); };
    // value x of row i into every CTA's copy of v; lanes p of P share the copies
    auto emit = [&](dd_t *v, int i, dd_t x, int p, int P) {
        if (i >= n) return;
        if (SMEM) {
            for (int d = p; d < R; d += P) *cl.map_shared_rank(reinterpret_cast<double2 *>(v) + i, d) = make_double2(x.hi, x.lo);
        } else if (p == 0) {
            __stcg(reinterpret_cast<double2 *>(v) + i, make_double2(x.hi, x.lo));
        }
    };
    // few own chunks: 2, 4, 8 or 16 warps share a chunk's terms
    int lp = 0;
    while (nch > 0 && (2 << lp) * nch <= LZ_WARPS) ++lp;
    const int part = warp & ((1 << lp) - 1);
    // one product: rows of this CTA's chunks, summed over the parts, to v
    // (wl when v is null)
    auto product = [&](auto &&chunk, dd_t *v) {
        for (int s = warp >> lp; s < nch; s += LZ_WARPS >> lp) {
            const dd_t t = chunk((rank + R * s) * LZ_CHUNK);
            const int row = lane & 7, p = lane >> 3;
            if (lp > 0) {
                if (p == 0) S.psum[((s * LZ_CHUNK + row) << lp) + part] = t;
            } else if (v) {
                emit(v, (rank + R * s) * LZ_CHUNK + row, t, p, 4);
            } else if (p == 0) {
                wl[s * LZ_CHUNK + row] = t;
            }
        }
        if (lp > 0) {
            __syncthreads();
            const int live = nown << lp; // at most 128, whole groups of 2^lp lanes
            if (tid < live) {
                const int left = live - warp * 32;
                const unsigned mask = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
                dd_t t = S.psum[tid];
                for (int m = 1; m < 1 << lp; m <<= 1)
                    t = dd_add(t, dd_make(__shfl_xor_sync(mask, t.hi, m), __shfl_xor_sync(mask, t.lo, m)));
                const int s = tid >> lp, p = tid & ((1 << lp) - 1);
                if (v)
                    emit(v, row_of(s), t, p, 1 << lp);
                else if (p == 0)
                    wl[s] = t;
            }
        }
    };
    // sum of the CTAs' parts, the same in every thread
    auto gather = [&](const dd_t *p) {
        dd_t t = lane < R ? p[lane] : dd_zero();
        for (int m = 1; m < R; m <<= 1) t = dd_add(t, shfl_xor_dd(t, m));
        return shfl_dd(t, 0);
    };

    for (int i = tid; i < n; i += LZ_THREADS) {
        if (SMEM || rank == 0) {
            st_dd(q + i, dd_zero());
            st_dd(tmp + i, dd_from(1.0));
        }
    }
    for (int s = tid; s < nown; s += LZ_THREADS) ql[s] = dd_zero();
    dd_t mn = dd_from(1.0e+51), mn_old = dd_from(1.0e+52), err = dd_from(1.0e+10), beta = dd_sqrt(dd_from((double)n));
    dd_t value = dd_div(dd_from(1.0), beta); // 1 / beta
    const dd_t sqn10 = dd_add_d(beta, 10.0);
    const dd_t sqn9 = dd_sqrt(dd_add_d(dd_from((double)n), 9.0));
    cl.sync();
    int k = 0, kk = 0;
    while (true) {
        const bool c1 = dd_gt(dd_abs(dd_sub(mn, mn_old)), dd_add_d(dd_mul_d(dd_abs(mn), 1.0e-5), 1.0e-8));
        const bool c2 = dd_gt(dd_abs(dd_mul(err, beta)), dd_add_d(dd_mul_d(dd_abs(mn), 1.0e-2), 1.0e-4));
        if (!(k < n && k < LZ_KMAX && d_lt_dd((double)k, sqn10) && dd_gt_d(beta, 1.0e-16) && (c1 || c2))) break;
        if (tid == 0 && k > 0) S.ioff[k - 1] = value;
        // qold = q; q = r * value (Rcopy + Rscal)
        for (int s = tid; s < nown; s += LZ_THREADS) {
            const int i = row_of(s);
            if (i < n && k > 0) {
                const double2 x = lz_ld<SMEM>(q, i);
                ql[s] = dd_make(x.x, x.y);
            }
        }
        if (SMEM) {
            __syncthreads();
            for (int i = tid; i < n; i += LZ_THREADS) st_dd(q + i, dd_mul(value, ld_dd(tmp + i)));
            __syncthreads();
        } else {
            for (int s = tid; s < nown; s += LZ_THREADS) {
                const int i = row_of(s);
                if (i < n) {
                    const double2 x = __ldcg(reinterpret_cast<const double2 *>(tmp) + i);
                    emit(q, i, dd_mul(value, dd_make(x.x, x.y)), 0, 1);
                }
            }
            cl.sync();
        }
        // w = L^T q (Rtrmv "Lower","Transpose")
        product([&](int i0) { return lz_rows<LZ_LOWER_T, SMEM>(L, n, i0, part, lp, q); }, w);
        cl.sync();
        // tmp = X w (Rgemv "N", alpha 1, beta 0)
        product([&](int i0) { return lz_rows<LZ_FULL, SMEM>(X, n, i0, part, lp, w); }, tmp);
        cl.sync();
        // w = L tmp (Rtrmv "Lower","NoTranspose"): own rows, and their part of
        // alpha = q.w
        product([&](int i0) { return lz_rows<LZ_LOWER, SMEM>(L, n, i0, part, lp, tmp); }, nullptr);
        __syncthreads();
        if (warp == 0) {
            DotAcc acc;
            for (int s = lane; s < nown; s += 32) {
                const int i = row_of(s);
                if (i < n) acc.term(lz_ld<SMEM>(q, i), make_double2(wl[s].hi, wl[s].lo));
            }
            const dd_t t = warp_sum_dd(acc.value());
            if (lane < R) *cl.map_shared_rank(&S.pa[rank], lane) = t;
        }
        cl.sync();
        const dd_t alpha = gather(S.pa);
        if (tid == 0) S.diag[k] = alpha;
        // r = w - alpha q - beta qold (Rcopy, Raxpy, Raxpy), own rows, and
        // their part of r.r
        if (warp == 0) {
            const dd_t ma = dd_neg(alpha), mb = dd_neg(beta);
            DotAcc acc;
            for (int s = lane; s < nown; s += 32) {
                const int i = row_of(s);
                if (i >= n) continue;
                const double2 qi = lz_ld<SMEM>(q, i);
                dd_t ri = dd_acc(wl[s], dd_mul(ma, dd_make(qi.x, qi.y)));
                ri = dd_acc(ri, dd_mul(mb, ql[s]));
                acc.term(make_double2(ri.hi, ri.lo), make_double2(ri.hi, ri.lo));
                emit(tmp, i, ri, 0, 1);
            }
            const dd_t t = warp_sum_dd(acc.value());
            if (lane < R) *cl.map_shared_rank(&S.pr[rank], lane) = t;
        }
        cl.sync();
        {
            // 1/beta and beta from one reciprocal square root and a Newton step
            const dd_t rr = gather(S.pr);
            const double x = rsqrt(rr.hi);
            const dd_t t = dd_mul(rr, dd_sqr_d(x));
            value = dd_add_dd_exact(x, 0.5 * x * ((1.0 - t.hi) - t.lo));
            beta = dd_mul(rr, value);
            if (!(rr.hi > 0.0)) beta = dd_sqrt(rr); // zero or not a number: the loop ends
        }
        if (tid == 0) S.off[k] = beta;
        // checkpoint: kk >= sqrt(k) || k == n-1 || k > sqrt(n+9)
        if (dd_le_d(dd_sqrt(dd_from((double)k)), (double)kk) || k == n - 1 || d_gt_dd((double)k, sqn9)) {
            kk = 0;
            mn_old = mn;
            tri_min_eigenpair<LZ_KMAX, LZ_WARPS>(k + 1, S.diag, S.off, S.ioff, S.tri, mn, err);
        }
        ++k;
        ++kk;
    }
    if (rank == 0 && tid == 0) out[cid] = dd_sub(mn, dd_abs(dd_mul(err, beta)));
}

// CTAs of a block's cluster.  A step's 2 n^2 terms are FP64-bound on one SM
// from a few dozen rows on and read n^2 dd values of X and n^2 of L through
// the SMs' L2 ports; four cluster barriers a step cost about 0.2 us each.
// Whole runs of L L L^T on a B200, us, for 2 / 4 / 8 / 16 CTAs: n = 30: 252 /
// 258 / 261 / 268; n = 64: 291 / 285 / 291 / 299; n = 100: 406 / 350 / 338 /
// 343; n = 150: 676 / 518 / 439 / 408; n = 200: 903 / 662 / 520 / 476; n =
// 500: 3420 / 2207 / 1372 / 990 (one CTA: 6562).  With many blocks the launch
// fills the GPU by itself.
int lanczos_cluster(long n, int blocks, int most) {
    int R = n <= 64 ? 2 : n <= 96 ? 4 : n <= 144 ? 8 : 16;
    R = std::min(R, most);
    while (R > 1 && (long)R * blocks > 148) R /= 2;
    return R;
}

size_t lanczos_smem(long n, int R, bool vectors) {
    const long chunks = (n + LZ_CHUNK - 1) / LZ_CHUNK, own = (chunks + R - 1) / R * LZ_CHUNK;
    return sizeof(LanczosShared) + sizeof(dd_t) * (2 * own + (vectors ? 3 * n : 0));
}

} // namespace

void launch_lanczos(cudaStream_t st, const int *ids, int nb, int nsp, long maxn, const int *sizes, const long *off, const dd_t *L, const dd_t *D,
                    const dd_t *L2, const dd_t *D2, dd_t *work, long work_stride, dd_t *out) {
    constexpr size_t SMEM_MAX = 227 * 1024;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    // most CTAs a cluster may have here (more than 8 is the device's choice)
    static thread_local int most[64] = {};
    if (most[dev & 63] == 0) {
        for (auto *f : {lanczos_kernel<true>, lanczos_kernel<false>}) {
            CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
            CK(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        }
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(LZ_CLUSTER);
        q.blockDim = dim3(LZ_THREADS);
        q.dynamicSmemBytes = SMEM_MAX;
        cudaLaunchAttribute a[1];
        a[0].id = cudaLaunchAttributeClusterDimension;
        a[0].val.clusterDim.x = LZ_CLUSTER;
        a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
        q.attrs = a;
        q.numAttrs = 1;
        int clusters = 0;
        const bool ok = cudaOccupancyMaxActiveClusters(&clusters, lanczos_kernel<true>, &q) == cudaSuccess && clusters >= 1;
        if (!ok) cudaGetLastError();
        most[dev & 63] = ok ? LZ_CLUSTER : 8;
    }
    // The split of the sums, and so a value's last bits, follow the cluster's
    // size; sized for two spaces in either case, so that an eigenvalue asked for
    // alone is the one that the solver's launch over both spaces gives.
    // A CTA's own rows of two vectors are in shared memory in either form, so a
    // large block among many small ones needs a larger cluster than their number
    // asks for (one CTA holds 6200 rows).
    int R = lanczos_cluster(maxn, 2 * nb, most[dev & 63]);
    while (R < most[dev & 63] && lanczos_smem(maxn, R, false) > SMEM_MAX) R *= 2;
    const bool smem = lanczos_smem(maxn, R, true) <= SMEM_MAX;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nb * nsp * R));
    cfg.blockDim = dim3(LZ_THREADS);
    cfg.dynamicSmemBytes = lanczos_smem(maxn, R, smem);
    cfg.stream = st;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeClusterDimension;
    a[0].val.clusterDim.x = (unsigned)R;
    a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    CK(cudaLaunchKernelEx(&cfg, smem ? lanczos_kernel<true> : lanczos_kernel<false>, ids, nb, sizes, off, L, D, L2, D2, work, work_stride, out));
    CK_LAUNCH();
}

// Smallest eigenvalue of the lower triangle of an n x n symmetric M
// (n <= 32): Householder tridiagonalisation, then tri_eig.cuh.  One warp per
// block, row i on lane i, A in shared memory; the reflectors' sums go over
// the lanes (a butterfly of five exchanges), the products with A are one
// compensated dot a lane.  A latency chain of 18 reflections at n = 20: 82 us
// with the two products that form M; 235 us when lane 0 summed in sequence
// and a dd Sturm multisection followed.
__global__ void __launch_bounds__(32) small_min_eig_kernel(const int *blk_ids, const int *sizes, const long *off, const dd_t *Msp, dd_t *out) {
    __shared__ dd_t A[32][33];
    __shared__ dd_t v[32], w[32], d[32], e[32], ie[32];
    __shared__ TriWork<32, 1> tri;
    const int lane = threadIdx.x;
    const int b = blk_ids[blockIdx.x];
    const int n = sizes[b];
    const dd_t *M = Msp + off[b];
    for (int j = 0; j < n; ++j)
        if (lane >= j && lane < n) {
            const dd_t x = ld_dd(M + lane + (long)n * j);
            A[lane][j] = x;
            A[j][lane] = x;
        }
    __syncwarp();
    for (int k = 0; k + 2 < n; ++k) {
        const bool in = lane > k && lane < n;
        const dd_t x = in ? A[lane][k] : dd_zero();
        const dd_t nrm = dd_sqrt(warp_sum_dd(dd_mul(x, x)));
        if (dd_is_zero(nrm)) continue;
        // v = x - alpha e_{k+1} with alpha = -sign(x_{k+1}) |x|, and
        // v.v = 2 |x| (|x| + |x_{k+1}|)
        const dd_t x1 = A[k + 1][k];
        const dd_t alpha = x1.hi < 0.0 ? nrm : dd_neg(nrm);
        const dd_t tau = dd_div(dd_from(1.0), dd_mul(nrm, dd_add(nrm, dd_abs(x1))));
        const dd_t vi = lane == k + 1 ? dd_sub(x1, alpha) : x;
        v[lane] = vi;
        __syncwarp();
        // p = tau A v (row i on lane i; row k too: it takes the reflection)
        dd_t p = dd_zero();
        if (lane >= k && lane < n) {
            DotAcc acc;
            for (int j = k + 1; j < n; ++j) acc.term(make_double2(A[lane][j].hi, A[lane][j].lo), make_double2(v[j].hi, v[j].lo));
            p = dd_mul(tau, acc.value());
        }
        // K = tau/2 v^T p ; w = p - K v
        const dd_t K = dd_mul(dd_mul_d(tau, 0.5), warp_sum_dd(dd_mul(vi, p)));
        const dd_t wi = dd_sub(p, dd_mul(K, vi));
        w[lane] = wi;
        __syncwarp();
        // A -= v w^T + w v^T on rows and columns k .. n-1 (row i on lane i)
        if (lane >= k && lane < n) {
            const double2 nv = make_double2(-vi.hi, -vi.lo), nw = make_double2(-wi.hi, -wi.lo);
            for (int j = k; j < n; ++j) {
                DotAcc acc;
                acc.s = A[lane][j].hi;
                acc.e = A[lane][j].lo;
                acc.term(nv, make_double2(w[j].hi, w[j].lo));
                acc.term(nw, make_double2(v[j].hi, v[j].lo));
                A[lane][j] = acc.value();
            }
        }
        __syncwarp();
    }
    if (lane < n) {
        d[lane] = A[lane][lane];
        if (lane + 1 < n) {
            e[lane] = A[lane + 1][lane];
            ie[lane] = dd_div(dd_from(1.0), e[lane]);
        }
    }
    __syncwarp();
    dd_t lam, last;
    tri_min_eigenpair<32, 1>(n, d, e, ie, tri, lam, last);
    if (lane == 0) out[blockIdx.x] = lam;
}

// The small blocks (n <= 20) of one space: DLS2 = D L^T (Rgemm "N","T"),
// DLS1 = L DLS2 (Rgemm "N","N"), then each block's smallest eigenvalue to
// res[0 ..) in block order.
static void small_blocks(Context &c, const Space &L, const Space &D, const std::vector<int> &small, dd_t *res) {
    cudaStream_t st = c.stream;
    for (const BlockRun &r : c.runs) {
        if (r.n > 20) continue;
        const int n = r.n, l = r.first;
        const long nn = (long)n * n;
        gemm(st, 'N', 'T', GEMM_STORE, n, n, n, D.blk(c.off, l), n, nn, L.blk(c.off, l), n, nn, c.W2.blk(c.off, l), n, nn, r.count, false);
        gemm(st, 'N', 'N', GEMM_STORE, n, n, n, L.blk(c.off, l), n, nn, c.W2.blk(c.off, l), n, nn, c.W1.blk(c.off, l), n, nn, r.count, false);
    }
    small_min_eig_kernel<<<(unsigned)small.size(), 32, 0, st>>>(c.eig_ids_small.p, c.d_sizes.p, c.d_off.p, c.W1.buf.p, res);
    CK_LAUNCH();
}

// min over the blocks of lambda_min(L D L^T) for nsp spaces (1 or 2): the
// big blocks' Lanczos of all spaces in one launch; results per space in
// block order, then the minimum as the reference takes it.
static void min_eig_spaces(Context &c, int nsp, const Space *L[2], const Space *D[2], dd_t out[2]) {
    cudaStream_t st = c.stream;
    PROF_SCOPE("min_eig", st);
    std::vector<int> big, small;
    for (int l = 0; l < c.nSDP; ++l) (c.sizes[l] > 20 ? big : small).push_back(l);
    static_assert(LZ_KMAX >= 64, "Lanczos step bound");
    if (c.eig_ids_big.n != big.size() || c.eig_ids_small.n != small.size() || c.eig_ids_gen != c.upload_gen) {
        c.eig_ids_big.upload(big, st);
        c.eig_ids_small.upload(small, st);
        c.eig_ids_gen = c.upload_gen;
    }
    const size_t nb = big.size(), ns = small.size();
    // result slots: space s at s * nSDP: big blocks first, then the small
    dd_t *res = c.scal.p;
    if (nb > 0) {
        long maxn = 0;
        for (int l : big) maxn = std::max<long>(maxn, c.sizes[l]);
        c.eig_work.alloc(LZ_WORK * maxn * nb * nsp);
        // the two spaces' clusters write slots 0 .. 2 nb - 1; spread below
        launch_lanczos(st, c.eig_ids_big.p, (int)nb, nsp, maxn, c.d_sizes.p, c.d_off.p, L[0]->buf.p, D[0]->buf.p, L[nsp - 1]->buf.p,
                       D[nsp - 1]->buf.p, c.eig_work.p, LZ_WORK * maxn, res + 2 * c.nSDP);
    }
    for (int sp = 0; sp < nsp && ns > 0; ++sp) small_blocks(c, *L[sp], *D[sp], small, res + (size_t)sp * c.nSDP + nb);
    if (nb > 0) {
        for (int sp = 0; sp < nsp; ++sp)
            CK(cudaMemcpyAsync(res + (size_t)sp * c.nSDP, res + 2 * c.nSDP + sp * nb, sizeof(dd_t) * nb, cudaMemcpyDeviceToDevice, st));
    }
    std::vector<dd_t> h((size_t)nsp * c.nSDP);
    d2h(c, h.data(), res, sizeof(dd_t) * h.size());
    for (int sp = 0; sp < nsp; ++sp) {
        // blocks in order: big blocks' values first in the slots, then the small
        const dd_t *v = h.data() + (size_t)sp * c.nSDP;
        size_t bi = 0, si = 0;
        dd_t mn = dd_from(1.0e50);
        for (int l = 0; l < c.nSDP; ++l) {
            const dd_t x = (c.sizes[l] > 20) ? v[bi++] : v[nb + si++];
            if (dd_lt(x, mn)) mn = x;
        }
        out[sp] = mn;
    }
}

dd_t min_eig(Context &c, const Space &L, const Space &D) {
    const Space *Ls[2] = {&L, &L}, *Ds[2] = {&D, &D};
    dd_t out[2];
    min_eig_spaces(c, 1, Ls, Ds, out);
    return out[0];
}

void min_eig_pair(Context &c, const Space &L1, const Space &D1, const Space &L2, const Space &D2, dd_t &out1, dd_t &out2) {
    const Space *Ls[2] = {&L1, &L2}, *Ds[2] = {&D1, &D2};
    dd_t out[2];
    min_eig_spaces(c, 2, Ls, Ds, out);
    out1 = out[0];
    out2 = out[1];
}

} // namespace sddd
