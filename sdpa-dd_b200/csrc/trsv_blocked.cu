// Blocked dd triangular solves for the tensor-core split form.
//
// The split form's Cholesky factor of B is not the reference's bit pattern
// (its trailing updates round once per panel), so its solves need not keep
// Rtrsv's per-entry chain either.  Here the 64 x 64 diagonal blocks of L
// are inverted once per factorisation (trsv_diag_inverse, one CTA per
// block, all blocks at once), and a solve is a wavefront of 64-entry
// blocks in which no step divides or waits on a single entry:
//   'N'  v_c = b_c - sum_{p<c} L(c,p) x_p,   x_c = W_c v_c
//   'T'  v_c = b_c - sum_{p>c} L(p,c)^T x_p, x_c = W_c^T v_c   (W_c = L(c,c)^-1)
// followed by one step of iterative refinement against L(c,c) itself,
// x_c += W_c (v_c - L(c,c) x_c) (transposed for 'T'), which brings the
// block's solve to the accuracy of a substitution even where L(c,c) is far
// from orthogonal (the Schur matrix near the optimum).
// One cooperative launch per solve: CTA k owns blocks k, k + G, ... (in
// solve order).  For each of its blocks it streams the tiles L(c,p) (or
// L(p,c)) and finally W_c into shared memory with bulk copies (one copy per
// tile column of up to 1 KB, three tiles in flight, completion on an
// mbarrier), waits (bounded) for block p's entries, which carry the solve's epoch, and
// all 256 threads multiply: thread (r, q) sums every fourth product of row r
// (or column r), so the critical path per block is one tile and three triangular
// 64 x 64 products (W_c, L(c,c), W_c), each followed by a 4-way combination.
// L is read once per solve.  Right-hand sides go side by side (grid row y).
//
// What bounds a block is one SM's FP64 issue rate: 4096 products and sums in
// dd operations are 29 instructions each, 1.9k cycles.  So a thread's sum is
// a compensated one (Ogita, Rump, Oishi, "Accurate sum and dot product",
// SIAM J. Sci. Comput. 26, 2005): the high parts' products summed with their
// rounding errors collected beside (12 instructions a term, and a chain of
// one addition), rounded to a dd per thread.
// Measured, n = 5003: 426 us for one solve or two side by side; with dd sums of 16
// consecutive terms, all of W_c multiplied, the quarters' sums through shared memory
// and a flag per block 583; n = 9980 840, before 1144.
//
// Every wait is bounded (the solve's wait budget, 2 s by default); a CTA
// that gives up records the awaited block in the error word (read by
// trsv_check), waits (bounded) for its copies in flight and returns.
#include "blas.h"
#include "bulk.cuh"
#include "devops.cuh"
#include "prof.h"

namespace sddd {

namespace {

constexpr int TB = 64;           // block order
constexpr int TB_LD = 65;        // padded leading dimension of a tile in shared memory
constexpr int TB_STAGES = 3;     // tiles in flight per CTA
constexpr int TB_Q = 4;          // threads that share a row of a tile
constexpr int TB_THREADS = TB * TB_Q;
constexpr int TB_TILE = TB * TB_LD; // double2 per stage

struct TbShared {
    uint64_t bar[TB_STAGES];
    int fail;
    long fail_at; // the first tile not consumed when the CTA gave up
};
constexpr size_t TB_SMEM = sizeof(double2) * ((size_t)TB_STAGES * TB_TILE + 3 * TB) + 128;
static_assert(TB_SMEM <= 232448, "blocked solve: shared memory above the per-CTA limit");

struct TbArgs {
    const dd_t *L;
    long lda;
    const dd_t *W; // nblk tiles of TB x TB (leading dimension TB): L(c,c)^-1, lower
    int n, nblk, epoch, trans; // trans: 0 'N', 1 'T'
    dd_t *x;
    unsigned long long *xch; // published entries: TB_REC words each
    int *err;
    unsigned long long wait_ns;
    int withhold; // a block that is never published (-1: none)
    long ldx;     // between right-hand sides
};

// The k-th tile block c reads: 'N' L(c, k) for k < c, 'T' L(nblk-1-k, c)
// for k < nblk-1-c; then L(c,c) and W_c (ntiles = 'N' c + 2, 'T' nblk-c+1).  Column j of the tile (rows
// r0 .. r0+rows-1 of column c0 + j) goes to T + j * TB_LD.
struct TileSrc {
    const dd_t *base; // column 0, row 0
    long ld;          // between columns
    int rows, cols;
};

__device__ __forceinline__ TileSrc tb_tile(const TbArgs &a, int c, int k, int ntiles) {
    const int nbc = min(TB, a.n - c * TB);
    TileSrc s;
    if (k == ntiles - 1) {
        s.base = a.W + (long)c * TB * TB;
        s.ld = TB;
        s.rows = nbc;
        s.cols = nbc;
    } else if (k == ntiles - 2) {
        s.base = a.L + (long)c * TB + a.lda * (long)(c * TB);
        s.ld = a.lda;
        s.rows = nbc;
        s.cols = nbc;
    } else if (a.trans == 0) {
        s.base = a.L + (long)c * TB + a.lda * (long)(k * TB);
        s.ld = a.lda;
        s.rows = nbc;
        s.cols = TB; // p = k < c: a full block
    } else {
        const int p = a.nblk - 1 - k;
        s.base = a.L + (long)p * TB + a.lda * (long)(c * TB);
        s.ld = a.lda;
        s.rows = min(TB, a.n - p * TB);
        s.cols = nbc;
    }
    return s;
}

// Warp 0: the copies of one tile into stage buffer T (lane l copies
// columns l and l + 32).
__device__ __forceinline__ void tb_issue(const TileSrc &s, double2 *T, uint64_t *bar, int lane) {
    if (lane == 0) mbar_expect_tx(bar, (uint32_t)(s.rows * s.cols * (int)sizeof(double2)));
    __syncwarp();
    for (int j = lane; j < s.cols; j += 32) bulk_g2s(T + j * TB_LD, s.base + s.ld * (long)j, (uint32_t)(s.rows * sizeof(double2)), bar);
}

// Bounded wait on a stage's mbarrier (thread 0 only).
__device__ bool tb_wait_bar(uint64_t *bar, uint32_t parity, unsigned long long wait_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity))
        if (globaltimer_ns() - t0 > wait_ns) return false;
    return true;
}

__device__ __forceinline__ int tb_ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// A published entry: its four 32-bit words, each in the upper half of a 64-bit
// word whose lower half is the solve's epoch.  64-bit accesses are single, so a
// reader that finds the epoch in all four has the entry, without a fence and a
// second round trip behind a flag.
constexpr int TB_REC = 4;
static_assert((size_t)TB * TB_REC == TRSV_XCH_BLOCK, "published words of a block");
__device__ __forceinline__ void tb_publish(unsigned long long *rec, int epoch, dd_t v) {
    const unsigned long long e = (unsigned)epoch, h = (unsigned long long)__double_as_longlong(v.hi), l = (unsigned long long)__double_as_longlong(v.lo);
    const unsigned long long up = 0xffffffff00000000ull;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(rec), "l"((h & up) | e), "l"((h << 32) | e) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(rec + 2), "l"((l & up) | e), "l"((l << 32) | e) : "memory");
}
__device__ __forceinline__ bool tb_read(const unsigned long long *rec, int epoch, double2 &v) {
    unsigned long long a, b, c, d;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(rec) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "l"(rec + 2) : "memory");
    const unsigned e = (unsigned)epoch;
    const unsigned long long up = 0xffffffff00000000ull;
    v.x = __longlong_as_double((long long)((a & up) | (b >> 32)));
    v.y = __longlong_as_double((long long)((c & up) | (d >> 32)));
    return (unsigned)a == e && (unsigned)b == e && (unsigned)c == e && (unsigned)d == e;
}

// Bounded wait for an entry.  The error word and the clock are looked at once
// in a while only: either costs as much as a look at the entry.
__device__ bool tb_wait_entry(const TbArgs &a, const unsigned long long *rec, double2 &v) {
    for (int k = 0; k < 64; ++k)
        if (tb_read(rec, a.epoch, v)) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (!tb_read(rec, a.epoch, v)) {
        if (tb_ld_acquire(a.err) != 0 || globaltimer_ns() - t0 > a.wait_ns) return false;
        __nanosleep(20);
    }
    return true;
}

__device__ __forceinline__ dd_t sm_dd(const double2 *T, int i) {
    const double2 v = T[i];
    return dd_make(v.x, v.y);
}

__device__ __forceinline__ double2 tb_pack(dd_t v) { return make_double2(v.hi, v.lo); }

// A compensated sum of dd products: s + e + f, e the sum of the rounding errors
// of s, f that of the products' low parts; folded every eight terms, so that
// e and f stay an ulp or two of s (folded every tile only, the solve's error on
// a factor of condition 1e8 was 12 % above that of dd sums).
struct TbSum {
    double s = 0.0, e = 0.0, f = 0.0;
    __device__ __forceinline__ void add(double2 x, double2 y) {
        const double p = __dmul_rn(x.x, y.x);
        const double pe = __fma_rn(x.y, y.x, __fma_rn(x.x, y.y, __fma_rn(x.x, y.x, -p)));
        double t;
        s = ddm::two_sum(s, p, t);
        e = __dadd_rn(e, t);
        f = __dadd_rn(f, pe);
    }
    // s the rounded sum, e the rest
    __device__ __forceinline__ void fold() {
        double t;
        e = ddm::two_sum(e, f, f);
        s = ddm::two_sum(s, e, t);
        e = __dadd_rn(t, f);
        f = 0.0;
    }
    // the sum over a row's lanes
    __device__ __forceinline__ void join() {
#pragma unroll
        for (int m = 32 / TB_Q; m < 32; m *= 2) {
            double t, u;
            s = ddm::two_sum(s, __shfl_xor_sync(0xffffffffu, s, m), t);
            e = ddm::two_sum(e, __shfl_xor_sync(0xffffffffu, e, m), u);
            f = __dadd_rn(__dadd_rn(f, __shfl_xor_sync(0xffffffffu, f, m)), u);
            e = ddm::two_sum(e, t, u);
            f = __dadd_rn(f, u);
        }
    }
    __device__ __forceinline__ dd_t dd() const {
        TbSum w = *this;
        w.fold();
        double l;
        const double h = ddm::fast_two_sum(w.s, w.e, l);
        return dd_make(h, l);
    }
};

// Thread (r, q)'s part of row r of M y ('N') or of column r of M^T y ('T'):
// the terms t2 = q, q + TB_Q, .. of [lo, hi).
__device__ __forceinline__ void tb_dot(TbSum &w, const double2 *M, const double2 *y, int r, int q, int lo, int hi, int trans) {
    int t2 = q + (max(lo - q, 0) + TB_Q - 1) / TB_Q * TB_Q;
    const double2 *m = trans == 0 ? M + r : M + r * TB_LD;
    const int ld = trans == 0 ? TB_LD : 1;
#pragma unroll
    for (int half = 1; half <= 2; ++half) {
        const int end = min(hi, half * TB / 2);
#pragma unroll 4
        for (; t2 < end; t2 += TB_Q) w.add(m[t2 * ld], y[t2]);
        w.fold();
    }
}

// A row (or column) of a tile and the residue of its other index: a row's TB_Q
// lanes lie in one warp, and eight neighbouring lanes read eight neighbouring
// rows (columns), so different banks.
__device__ __forceinline__ int tb_row(int warp, int lane) { return 8 * warp + (lane & 7); }
__device__ __forceinline__ int tb_residue(int lane) { return lane >> 3; }
static_assert(TB_Q == 4, "eight rows a warp");

// Entry r of M y ('N') or M^T y ('T') for a lower triangular M (M(i,j), i >= j)
// of order nb, in the row's lanes.
__device__ __forceinline__ dd_t tb_lower(const double2 *M, const double2 *y, int r, int q, int nb, int trans) {
    TbSum w;
    if (r < nb) tb_dot(w, M, y, r, q, trans ? r : 0, trans ? nb : r + 1, trans);
    w.join();
    return w.dd();
}

__global__ void __launch_bounds__(TB_THREADS, 1) trsv_blocked_kernel(TbArgs a) {
    extern __shared__ __align__(128) double2 tb_sm[];
    double2 *tiles = tb_sm;                      // TB_STAGES x TB_TILE
    double2 *xs = tiles + TB_STAGES * TB_TILE;   // TB: x of block p, then v of block c
    double2 *x0 = xs + TB;                       // TB: W_c v
    double2 *rs = x0 + TB;                       // TB: v - L(c,c) x0
    TbShared &S = *reinterpret_cast<TbShared *>(rs + TB);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = tb_row(warp, lane), q = tb_residue(lane);
    a.x += a.ldx * blockIdx.y;
    a.xch += (long)a.nblk * TB * TB_REC * blockIdx.y;
    if (tid == 0) {
        for (int s = 0; s < TB_STAGES; ++s) mbar_init(&S.bar[s], 1);
        S.fail = 0;
        mbar_init_fence();
    }
    __syncthreads();
    long g = 0;        // tiles consumed by this CTA (stage and parity)
    long issued = 0;   // tiles whose copies this CTA issued
    for (int k = blockIdx.x; k < a.nblk; k += gridDim.x) {
        const int c = a.trans == 0 ? k : a.nblk - 1 - k;
        const int nbc = min(TB, a.n - c * TB);
        const int ntiles = a.trans == 0 ? c + 2 : a.nblk - c + 1;
        if (warp == 0)
            for (int t = 0; t < TB_STAGES && t < ntiles; ++t) {
                const int st = (int)((g + t) % TB_STAGES);
                tb_issue(tb_tile(a, c, t, ntiles), tiles + st * TB_TILE, &S.bar[st], lane);
            }
        issued = g + min(TB_STAGES, ntiles);
        TbSum acc;
        const dd_t bc = r < nbc ? ld_dd(a.x + (long)c * TB + r) : dd_zero();
        bool failed = false; // (the shared word may be set again below: every thread keeps what it saw)
        for (int t = 0; t < ntiles - 2; ++t) {
            const long gt = g + t;
            const int st = (int)(gt % TB_STAGES);
            const double2 *T = tiles + st * TB_TILE;
            const int p = a.trans == 0 ? t : a.nblk - 1 - t; // block whose x this tile multiplies
            if (tid < TB) {
                // each lane of warps 0 and 1 waits for an entry of block p
                bool ok = true;
                int code = c + 1; // a tile of this block never landed
                if (tid == 0) ok = tb_wait_bar(&S.bar[st], (uint32_t)((gt / TB_STAGES) & 1), a.wait_ns);
                if (ok) {
                    code = p + 1; // the block waited for
                    double2 v = make_double2(0.0, 0.0);
                    if (p * TB + tid < a.n) ok = tb_wait_entry(a, a.xch + ((long)p * TB + tid) * TB_REC, v);
                    xs[tid] = v;
                }
                if (!ok) {
                    S.fail = 1;
                    S.fail_at = gt;
                    atomicCAS(a.err, 0, code);
                }
            }
            __syncthreads();
            failed = S.fail != 0;
            if (failed) break;
            // rows (or columns) r of block c
            if (r < nbc) tb_dot(acc, T, xs, r, q, 0, a.trans == 0 ? TB : min(TB, a.n - p * TB), a.trans);
            __syncthreads(); // stage st and xs are free again
            if (t + TB_STAGES < ntiles) {
                if (warp == 0) tb_issue(tb_tile(a, c, t + TB_STAGES, ntiles), tiles + st * TB_TILE, &S.bar[st], lane);
                issued = gt + TB_STAGES + 1;
            }
        }
        if (!failed) {
            // L(c,c) and W_c
            const long gl = g + ntiles - 2, gw = gl + 1;
            const double2 *Lc = tiles + (int)(gl % TB_STAGES) * TB_TILE, *Wc = tiles + (int)(gw % TB_STAGES) * TB_TILE;
            acc.join();
            if (tid == TB_THREADS - 1) {
                const bool ok = tb_wait_bar(&S.bar[gl % TB_STAGES], (uint32_t)((gl / TB_STAGES) & 1), a.wait_ns) &&
                                tb_wait_bar(&S.bar[gw % TB_STAGES], (uint32_t)((gw / TB_STAGES) & 1), a.wait_ns);
                if (!ok) {
                    S.fail = 1;
                    S.fail_at = gl;
                    atomicCAS(a.err, 0, c + 1);
                }
            }
            __syncthreads();
            failed = S.fail != 0;
            if (!failed) {
                // v = b_c - the products' sum
                const dd_t v = r < nbc ? dd_sub(bc, acc.dd()) : dd_zero();
                if (q == 0) xs[r] = tb_pack(v);
                __syncthreads();
                // x0 = W_c v ('N') or W_c^T v ('T')
                const dd_t y = tb_lower(Wc, xs, r, q, nbc, a.trans);
                if (q == 0) x0[r] = tb_pack(y);
                __syncthreads();
                // rs = v - L(c,c) x0 (lower triangle only: the strict upper
                // part of the tile holds the Schur matrix's own entries)
                const dd_t ly = tb_lower(Lc, x0, r, q, nbc, a.trans);
                if (q == 0) rs[r] = tb_pack(dd_sub(v, ly));
                __syncthreads();
                // x = x0 + W_c rs
                const dd_t x = dd_add(y, tb_lower(Wc, rs, r, q, nbc, a.trans));
                if (q == 0 && r < nbc) {
                    if (c != a.withhold) tb_publish(a.xch + ((long)c * TB + r) * TB_REC, a.epoch, x);
                    st_dd(a.x + (long)c * TB + r, x);
                }
                __syncthreads(); // the stages, xs, x0 and rs are free again
            }
        }
        if (failed) {
            // the copies issued but not consumed land (bounded waits)
            // before the CTA exits and its shared memory is reused
            if (tid == 0)
                for (long u = S.fail_at; u < issued; ++u) tb_wait_bar(&S.bar[u % TB_STAGES], (uint32_t)((u / TB_STAGES) & 1), a.wait_ns);
            __syncthreads();
            return;
        }
        g += ntiles;
    }
}

// W_c = L(c,c)^-1 for every diagonal block: one CTA per block; four lanes
// solve L(c,c) w = e_j for column j (rows j..nb-1, in order, into shared
// memory), each with every fourth term of a row, with the reciprocals of the
// pivots computed once.  n = 5003: 60 us; one thread a column 139, and with
// dd sums 156.
constexpr size_t TB_INV_SMEM = sizeof(double2) * (2 * (size_t)TB_TILE + TB);

__global__ void __launch_bounds__(TB_THREADS) trsv_diag_inverse_kernel(const dd_t *L, long lda, int n, dd_t *W) {
    extern __shared__ __align__(16) double2 inv_sm[];
    double2 *T = inv_sm;             // L(c,c), lower part
    double2 *Wt = inv_sm + TB_TILE;  // column j of the inverse at Wt + j * TB_LD
    double2 *rp = Wt + TB_TILE;      // 1 / L(i,i)
    const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int j = tb_row(tid >> 5, lane), q = tb_residue(lane);
    const int nb = min(TB, n - c * TB);
    const dd_t *D = L + (long)c * TB + lda * (long)(c * TB);
#pragma unroll 4
    for (int e = tid; e < TB * TB; e += TB_THREADS) {
        const int i = e % TB, col = e / TB;
        if (i < nb && col <= i) T[i + col * TB_LD] = *reinterpret_cast<const double2 *>(D + i + lda * (long)col);
    }
    __syncthreads();
    if (tid < nb) rp[tid] = tb_pack(dd_div(dd_make(1.0, 0.0), sm_dd(T, tid + tid * TB_LD)));
    __syncthreads();
    double2 *w = Wt + j * TB_LD;
    if (j < nb && q == 0) w[j] = rp[j];
    __syncwarp();
    // a warp's columns go down the rows together
    for (int i = tb_row(tid >> 5, 0) + 1; i < nb; ++i) {
        TbSum s;
#pragma unroll 4
        for (int k = j + q; k < i; k += TB_Q) s.add(T[i + k * TB_LD], w[k]);
        s.join();
        if (i > j && q == 0) w[i] = tb_pack(dd_mul(dd_neg(s.dd()), sm_dd(rp, i))); // w_i = -s / L(i,i)
        __syncwarp();
    }
    __syncthreads();
    // W_c column-major, leading dimension TB, zero above the diagonal and
    // outside the block; row-coalesced stores
    dd_t *Wc = W + (long)c * TB * TB;
    for (int e = tid; e < TB * TB; e += TB_THREADS) {
        const int i = e % TB, col = e / TB;
        st_dd(Wc + e, (col < nb && i < nb && i >= col) ? sm_dd(Wt, i + col * TB_LD) : dd_zero());
    }
}

} // namespace

void trsv_diag_inverse(cudaStream_t st, const dd_t *L, long lda, int n, dd_t *W) {
    if (n <= 0) return;
    PROF_SCOPE("trsv_diag_inverse", st);
    static thread_local bool attr[64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (!attr[dev & 63]) {
        CK(cudaFuncSetAttribute(trsv_diag_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TB_INV_SMEM));
        attr[dev & 63] = true;
    }
    trsv_diag_inverse_kernel<<<ceil_div(n, TB), TB_THREADS, TB_INV_SMEM, st>>>(L, lda, n, W);
    CK_LAUNCH();
}

void trsv_blocked(cudaStream_t st, char trans, const dd_t *L, long lda, int n, const dd_t *W, dd_t *x, TrsvSync &sync, int nrhs, long ldx) {
    if (n <= 0 || nrhs <= 0) return;
    if (trans != 'N' && trans != 'T') throw Error(ERR_ARG, "trsv_blocked: trans must be 'N' or 'T'");
    const int nblk = ceil_div(n, TB);
    if ((long)nblk * nrhs > sync.capacity || !sync.xch) throw Error(ERR_ARG, "trsv_blocked: progress flags hold fewer blocks than the solve needs");
    PROF_SCOPE("trsv", st);
    if (++sync.epoch <= 0) sync.epoch = 1;
    TbArgs a{L, lda, W, n, nblk, sync.epoch, trans == 'N' ? 0 : 1, x, sync.xch, sync.flags + sync.capacity, sync.wait_ns, sync.withhold, ldx};
    static thread_local int cap[64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int &cp = cap[dev & 63];
    if (cp == 0) {
        int sms = 0, per = 0;
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        CK(cudaFuncSetAttribute(trsv_blocked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TB_SMEM));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, trsv_blocked_kernel, TB_THREADS, TB_SMEM));
        if (per < 1) throw Error(ERR_CUDA, "trsv_blocked: the kernel does not fit on an SM");
        cp = per * sms;
    }
    // every CTA of the launch is resident: the right-hand sides share the SMs
    if (nrhs > cp) throw Error(ERR_ARG, "trsv_blocked: more right-hand sides than resident CTAs");
    const dim3 grid((unsigned)std::min(nblk, cp / nrhs), (unsigned)nrhs);
    void *args[] = {&a};
    CK(cudaLaunchCooperativeKernel((const void *)trsv_blocked_kernel, grid, TB_THREADS, args, TB_SMEM, st));
    CK_LAUNCH();
}

} // namespace sddd
