// Sparse Schur complement on the device (see sparse_chol.h).
//
// Storage.  The factor of the reordered B lives in the 64 x 64 tiles of its
// lower triangle that hold an entry of the symbolic factor; entry (a, b),
// a >= b, is the reference's sparse_bMat entry of row b, column a
// (Newton::initialize_sparse_bMat, sdpa_newton.cpp:225-340).  Each tile
// carries 64 structure words (word j: the rows of column j that belong to
// the symbolic factor), so that every kernel applies exactly the updates the
// reference applies and no other.
//
// Factor (Lal::getCholesky(SparseMatrix&, int*), sdpa_linear.cpp:353-395).
// Per pivot b in ascending order the reference sets d_b = 1 / sqrt(B(b,b))
// (0 when B(b,b) < 0), scales column b by it ("*="), then for every pair
// r <= a of struct(b) subtracts L(r,b) * L(a,b) from entry (a, r).  Each
// entry thus sees its updates in ascending pivot order, one dd multiply and
// one dd subtract each, and is scaled once, when its column becomes the
// pivot.  Here, per panel J of 64 pivots:
//   sp_panel_kernel   one CTA for the diagonal tile of column block J and two
//                     per tile below: every CTA factors the diagonal tile
//                     (pivots in order, the next column's pivot chain beside
//                     the other columns' updates), and the others carry half
//                     a tile below with the same pivots;
//   sp_update_kernel  every tile (I, K), K > J, that some column of J
//                     reaches in both I and K: entry (a, r) -= L(r,b) L(a,b)
//                     for the columns b of J ascending, where both are in
//                     the structure.
// Every entry keeps the reference's chain of operations, so the factor is
// the reference's bit for bit.
//
// Solves (Lal::solveSystems(Vector&, SparseMatrix&, Vector&),
// sdpa_linear.cpp:654-810, the loop that is compiled): forward over the
// entries in storage order, x(b) *= d_b at the diagonal and x(a) -= L(a,b)
// x(b) below it; backward in reverse storage order, x(b) -= L(a,b) x(a) for
// a descending, then x(b) *= d_b.  One cooperative launch per direction:
// CTA c owns row block c (forward) or the mirror order (backward), walks
// only the tiles of its row (column) block, and waits for the blocks it
// reads through per-block flags with a bounded wait, as the dense
// triangular solves do.
#include "sparse_chol.h"

#include <algorithm>

#include "fastdiv.cuh"
#include "prof.h"

namespace sddd {

constexpr int SPL = SP_T + 1; // padded leading dimension in shared memory
constexpr int SP_THREADS = 256;
constexpr int SP_UPD_SPLIT = 4; // CTAs per trailing-update tile (16 columns each)
constexpr size_t SP_TILE_SMEM = sizeof(double2) * SP_T * SPL;
constexpr size_t SP_TWO_TILES = 2 * SP_TILE_SMEM;
constexpr size_t SP_SOLVE_SMEM = 2 * SP_TILE_SMEM + 2 * sizeof(double2) * SP_T;

__device__ __forceinline__ bool bit64(unsigned long long w, int i) { return (w >> i) & 1ull; }
__device__ __forceinline__ dd_t sm_dd(const double2 *S, int i, int j) {
    const double2 v = S[i + SPL * j];
    return dd_make(v.x, v.y);
}
__device__ __forceinline__ void sm_st(double2 *S, int i, int j, dd_t v) { S[i + SPL * j] = make_double2(v.hi, v.lo); }

// Tile (contiguous 64 x 64, column-major) into shared memory with leading
// dimension 65: threads [t0, t0 + nt) put their 16-byte copies in flight
// and wait for them; the caller's barrier publishes the tile.
__device__ __forceinline__ void sp_load_tile(double2 *S, const dd_t *T, int t0, int nt) {
    for (int e = t0; e < SP_T * SP_T; e += nt) {
        const int i = e & (SP_T - 1), j = e >> 6;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(S + i + SPL * j)), "l"(T + e) : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void sp_store_tile(dd_t *T, const double2 *S, int t0, int nt) {
    for (int e = t0; e < SP_T * SP_T; e += nt) {
        const int i = e & (SP_T - 1), j = e >> 6;
        *reinterpret_cast<double2 *>(T + e) = S[i + SPL * j];
    }
}

// ------------------------------------------------------------ entries
// Tile entries from B through the order: (a, b) -> B(order[a], order[b])
// for the entries of the structure, zero elsewhere.
__global__ void sp_gather_B_kernel(const dd_t *B, int m, const int *order, const int *tIJ, const unsigned long long *mask, dd_t *tiles) {
    const int t = blockIdx.x;
    const int I = tIJ[2 * t], J = tIJ[2 * t + 1];
    for (int e = threadIdx.x; e < SP_T * SP_T; e += blockDim.x) {
        const int i = e & (SP_T - 1), j = e >> 6;
        const int a = I * SP_T + i, b = J * SP_T + j;
        dd_t v = dd_zero();
        if (a < m && b < m && bit64(mask[(long)t * SP_T + j], i)) v = ld_dd(B + order[a] + (long)m * order[b]);
        st_dd(tiles + (long)t * SP_T * SP_T + e, v);
    }
}

// Entries of the reference layout into the (zeroed) tiles, and back.
__global__ void sp_scatter_kernel(const dd_t *vals, const int *ent_b, const int *ent_a, long nnz, const int *tile_of, int nblk, dd_t *tiles) {
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= nnz) return;
    const int b = ent_b[q], a = ent_a[q];
    const int t = tile_of[a / SP_T + (long)nblk * (b / SP_T)];
    st_dd(tiles + (long)t * SP_T * SP_T + (a % SP_T) + SP_T * (b % SP_T), ld_dd(vals + q));
}
__global__ void sp_gather_kernel(const dd_t *tiles, const int *ent_b, const int *ent_a, long nnz, const int *tile_of, int nblk, dd_t *vals) {
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= nnz) return;
    const int b = ent_b[q], a = ent_a[q];
    const int t = tile_of[a / SP_T + (long)nblk * (b / SP_T)];
    st_dd(vals + q, ld_dd(tiles + (long)t * SP_T * SP_T + (a % SP_T) + SP_T * (b % SP_T)));
}

// ------------------------------------------------------------ panel
// CTA 0: the diagonal tile of panel J; CTA 1 + 2 k + h: the diagonal tile
// again (identical arithmetic) and rows 32 h .. 32 h + 31 of below-diagonal
// tile col_tiles[k].  Every CTA reads the unfactored diagonal tile at its
// start, so the factored one is written back by the CTA that finishes last
// (counted in done[J], which it resets for the next factorisation).
// Step c (one barrier): warp 0 publishes column c, the other warps apply its
// update to columns c+2.. (a column a warp at a time, rows over the lanes)
// while warp 0 takes column c+1 through it in registers and forms, in all its
// lanes, the next diagonal entry and its 1/sqrt; so the chain of pivots (a
// square root and reciprocal, a scaling, a product and a subtraction a column)
// runs beside the bulk of the updates, alone on its SM sub-partition (warps 4,
// 8, .. have no work), and every entry still sees pivot k's update before
// pivot k+1's.
// Chain of 200 blocks of order 20: 46 us a panel; with a whole tile below
// a CTA, the column through shared memory between its steps and the plain
// root and quotient on lane 0 75.
constexpr int SP_PANEL_THREADS = 512;
constexpr int SPH = SP_T / 2, SPHL = SPH + 1; // rows of a half tile, its leading dimension
constexpr size_t SP_PANEL_SMEM = SP_TILE_SMEM + sizeof(double2) * SPHL * SP_T;
__global__ void __launch_bounds__(SP_PANEL_THREADS) sp_panel_kernel(dd_t *tiles, const unsigned long long *mask, int m, int J, int diag_t,
                                                                    const int *col_tiles, int *done) {
    extern __shared__ double2 sp_sm[];
    double2 *D = sp_sm;
    double2 *U = sp_sm + SP_T * SPL; // used only when the CTA has rows below (ut >= 0, mu != 0)
    __shared__ unsigned long long md[SP_T];
    __shared__ uint32_t mu[SP_T];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = min(SP_T, m - J * SP_T);
    const int ut = blockIdx.x > 0 ? col_tiles[(blockIdx.x - 1) / 2] : -1;
    const int u0 = (blockIdx.x - 1) % 2 * SPH;
    dd_t *Ug = tiles + (long)max(ut, 0) * SP_T * SP_T + max(u0, 0);
    if (ut >= 0)
        for (int e = tid; e < SPH * SP_T; e += SP_PANEL_THREADS) {
            const int i = e % SPH, j = e / SPH;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(U + i + SPHL * j)), "l"(Ug + i + SP_T * j) : "memory");
        }
    sp_load_tile(D, tiles + (long)diag_t * SP_T * SP_T, tid, blockDim.x);
    if (tid < SP_T) {
        md[tid] = mask[(long)diag_t * SP_T + tid];
        mu[tid] = ut >= 0 ? (uint32_t)(mask[(long)ut * SP_T + tid] >> u0) : 0u;
    }
    __syncthreads();
    auto u_dd = [&](int j) {
        const double2 v = U[lane + SPHL * j];
        return dd_make(v.x, v.y);
    };
    auto u_st = [&](int j, dd_t v) { U[lane + SPHL * j] = make_double2(v.hi, v.lo); };
    const int ia = lane, ib = lane + 32; // this lane's rows of D
    if (warp == 0) {
        // column c through the pivots before it, and its diagonal entry in every lane
        dd_t xa = sm_dd(D, ia, 0), xb = sm_dd(D, ib, 0), xu = mu[0] ? u_dd(0) : dd_zero(), d = sm_dd(D, 0, 0);
        for (int c = 0; c < nb; ++c) {
            dd_t l, inv; // d_c = 1/sqrt(B(c,c)), 0 for a negative pivot
            if (!sqrt_rcp_fast(d, l, inv)) {
                if (dd_lt_d(d, 0.0)) inv = dd_zero();
                else sqrt_rcp_plain(d, l, inv);
            }
            const unsigned long long cc = md[c];
            const uint32_t uc = mu[c];
            const dd_t la = dd_muleq(xa, inv), lb = dd_muleq(xb, inv), lu = dd_muleq(xu, inv);
            const int cn = min(c + 1, SP_T - 1);
            const bool next = bit64(cc, cn);
            const dd_t ln = dd_make(__shfl_sync(0xffffffffu, cn < 32 ? la.hi : lb.hi, cn & 31), __shfl_sync(0xffffffffu, cn < 32 ? la.lo : lb.lo, cn & 31));
            if (ia > c && bit64(cc, ia)) sm_st(D, ia, c, la);
            if (ib > c && bit64(cc, ib)) sm_st(D, ib, c, lb);
            if (lane == 0) sm_st(D, c, c, inv);
            if (bit64(uc, lane)) u_st(c, lu);
            __syncthreads(); // column c is published, column c+1 has seen pivot c-1
            if (c + 1 >= nb) break;
            d = sm_dd(D, cn, cn);
            xa = sm_dd(D, ia, cn);
            xb = sm_dd(D, ib, cn);
            if (mu[cn]) xu = u_dd(cn);
            if (next) {
                d = dd_sub(d, dd_mul(ln, ln));
                const dd_t ya = dd_sub(xa, dd_mul(ln, la)), yb = dd_sub(xb, dd_mul(ln, lb)), yu = dd_sub(xu, dd_mul(ln, lu));
                if (ia >= cn && bit64(cc, ia)) xa = ya;
                if (ib >= cn && bit64(cc, ib)) xb = yb;
                if (bit64(uc, lane)) xu = yu;
            }
        }
    } else {
        const int h = (warp >> 2) * 3 + (warp & 3) - 1, nh = SP_PANEL_THREADS / 32 / 4 * 3;
        for (int c = 0; c < nb; ++c) {
            __syncthreads();
            if ((warp & 3) == 0) continue;
            const unsigned long long cc = md[c];
            const uint32_t uc = mu[c];
            const bool ba = bit64(cc, ia), bb = bit64(cc, ib), bu = bit64(uc, lane);
            const dd_t la = sm_dd(D, ia, c), lb = sm_dd(D, ib, c), lu = uc ? u_dd(c) : dd_zero();
            for (int r = c + 2 + h; r < nb; r += nh) {
                if (!bit64(cc, r)) continue;
                // entry (i, r) -= L(r,c) L(i,c)
                const dd_t lr = sm_dd(D, r, c);
                if (ba && ia >= r) sm_st(D, ia, r, dd_sub(sm_dd(D, ia, r), dd_mul(lr, la)));
                if (bb && ib >= r) sm_st(D, ib, r, dd_sub(sm_dd(D, ib, r), dd_mul(lr, lb)));
                if (bu) u_st(r, dd_sub(u_dd(r), dd_mul(lr, lu)));
            }
        }
    }
    __syncthreads();
    if (ut >= 0)
        for (int e = tid; e < SPH * SP_T; e += SP_PANEL_THREADS) {
            const int i = e % SPH, j = e / SPH;
            *reinterpret_cast<double2 *>(Ug + i + SP_T * j) = U[i + SPHL * j];
        }
    __shared__ int last;
    if (tid == 0) last = atomicAdd(done + J, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (last) {
        sp_store_tile(tiles + (long)diag_t * SP_T * SP_T, D, tid, blockDim.x);
        if (tid == 0) done[J] = 0;
    }
}

// ------------------------------------------------------------ update
// upd: (target, source (I, J), source (K, J)) per target; CTA q * 4 + p
// updates the 16 columns [16p, 16p + 16) of target q.
__global__ void __launch_bounds__(SP_THREADS) sp_update_kernel(dd_t *tiles, const unsigned long long *mask, const int *upd, int nbJ) {
    extern __shared__ double2 sp_sm[];
    double2 *SI = sp_sm;
    double2 *SK = sp_sm + SP_T * SPL;
    __shared__ unsigned long long mI[SP_T], mK[SP_T];
    const int tid = threadIdx.x;
    const int q = blockIdx.x / SP_UPD_SPLIT, part = blockIdx.x % SP_UPD_SPLIT;
    const int tt = upd[3 * q], sI = upd[3 * q + 1], sK = upd[3 * q + 2];
    const bool diag_target = sI == sK;
    sp_load_tile(SI, tiles + (long)sI * SP_T * SP_T, tid, blockDim.x);
    if (!diag_target) sp_load_tile(SK, tiles + (long)sK * SP_T * SP_T, tid, blockDim.x);
    if (tid < SP_T) {
        mI[tid] = mask[(long)sI * SP_T + tid];
        mK[tid] = mask[(long)sK * SP_T + tid];
    }
    __syncthreads();
    const double2 *SKp = diag_target ? SI : SK;
    dd_t *T = tiles + (long)tt * SP_T * SP_T;
    constexpr int COLS = SP_T / SP_UPD_SPLIT;
    for (int e = tid; e < SP_T * COLS; e += blockDim.x) {
        const int i = e & (SP_T - 1), k = part * COLS + (e >> 6);
        if (diag_target && i < k) continue;
        dd_t v = ld_dd(T + i + SP_T * k);
        for (int j = 0; j < nbJ; ++j)
            if (bit64(mI[j], i) && bit64(mK[j], k)) v = dd_sub(v, dd_mul(sm_dd(SKp, k, j), sm_dd(SI, i, j)));
        st_dd(T + i + SP_T * k, v);
    }
}

// ------------------------------------------------------------ solves
struct SpSolveArgs {
    const dd_t *tiles;
    const unsigned long long *mask;
    const int *tIJ, *row_ptr, *row_tiles, *col_ptr, *col_tiles, *diag;
    int m, nblk, epoch;
    dd_t *x;
    int *flags, *err;
    unsigned long long wait_ns;
    int withhold;
};

__device__ __forceinline__ int sp_ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sp_st_release(int *p, int v) { asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ unsigned long long sp_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Lane 0 waits (bounded) for block blk's flag; every lane gets the outcome.
__device__ bool sp_wait(const SpSolveArgs &a, int blk) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        const unsigned long long t0 = sp_ns();
        unsigned iter = 0;
        while (sp_ld_acquire(a.flags + blk) != a.epoch) {
            if (sp_ld_acquire(a.err) != 0 || ++iter > (1u << 26) || sp_ns() - t0 > a.wait_ns) {
                atomicCAS(a.err, 0, blk + 1);
                ok = 0;
                break;
            }
            if (iter > 64) __nanosleep(64);
        }
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
__device__ __forceinline__ dd_t sp_shfl(dd_t v, int src) {
    return dd_make(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
__device__ __forceinline__ dd_t sp_ldcg(const dd_t *p) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return dd_make(v.x, v.y);
}

// The diagonal tile by warp 0: entries lane and 32 + lane in v0, v1; steps s
// = 0 .. nb-1 (FWD) or nb-1 .. 0.  The chain x(s) -> x(s+1) runs in all lanes
// at once, the entries beyond are updated beside it; a step's operands are
// loaded a step ahead.
template <bool FWD> __device__ __forceinline__ void sp_diag(const double2 *T, const unsigned long long *msk, int nb, dd_t &v0, dd_t &v1) {
    const int lane = threadIdx.x & 31;
    auto el = [&](int e, int s) { return FWD ? sm_dd(T, e, s) : sm_dd(T, s, e); };
    auto in = [&](int e, int s) { return FWD ? bit64(msk[s], e) : bit64(msk[e], s); };
    auto entry = [&](int e) { return sp_shfl(e < 32 ? v0 : v1, e & 31); };
    const int inc = FWD ? 1 : -1, first = FWD ? 0 : nb - 1;
    auto at = [&](int q) { return first + inc * min(q, nb - 1); };
    int s = first, s1 = at(1);
    dd_t x = dd_muleq(entry(s), el(s, s)), w = entry(s1), fn = el(s1, s), f0 = el(lane, s), f1 = el(32 + lane, s), l = el(s1, s1);
    bool bn = in(s1, s), b0 = in(lane, s), b1 = in(32 + lane, s);
    for (int q = 0; q < nb; ++q) {
        const int s2 = at(q + 2);
        const dd_t gn = el(s2, s1), g0 = el(lane, s1), g1 = el(32 + lane, s1), ln = el(s2, s2);
        const bool cn = in(s2, s1), c0 = in(lane, s1), c1 = in(32 + lane, s1);
        const dd_t nv = dd_sub(w, dd_mul(fn, x)), n0 = dd_sub(v0, dd_mul(f0, x)), n1 = dd_sub(v1, dd_mul(f1, x));
        w = bn ? nv : w;
        v0 = lane == s ? x : (FWD ? lane > s : lane < s) && b0 ? n0 : v0;
        v1 = 32 + lane == s ? x : (FWD ? 32 + lane > s : 32 + lane < s) && b1 ? n1 : v1;
        x = dd_muleq(w, l);
        w = entry(s2);
        fn = gn, f0 = g0, f1 = g1, l = ln;
        bn = cn, b0 = c0, b1 = c1;
        s = s1;
        s1 = s2;
    }
}

// CTA b owns row blocks b, b + G, .. (forward) or the mirror (backward) and
// walks the tiles of its row (column) block in the order of the terms: when
// the block a tile multiplies is there, all threads form the tile's products
// in place, then two warps (an entry a lane) only subtract them, in the steps
// that some entry of the warp has, while the others bring the next tile.
// Chain of 200 blocks of order 20 (94 row blocks): 1.35 ms forward, 1.33
// backward; with one warp that multiplied, subtracted and scaled 1.73 and 1.72.
template <bool FWD> __global__ void __launch_bounds__(SP_THREADS) sp_solve_kernel(SpSolveArgs a) {
    extern __shared__ double2 sp_sm[];
    double2 *xs = sp_sm + 2 * SP_T * SPL, *vs = xs + SP_T;
    __shared__ unsigned long long msk[2][SP_T];
    __shared__ int fail;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) fail = 0;
    for (int k = blockIdx.x; k < a.nblk; k += gridDim.x) {
        const int c = FWD ? k : a.nblk - 1 - k, r0 = c * SP_T, nb = min(SP_T, a.m - r0);
        // tiles (c, J), J < c, ascending, or (I, c), I > c, descending; then
        // the diagonal tile
        const int *ptr = FWD ? a.row_ptr : a.col_ptr;
        const int q0 = ptr[c], q1 = ptr[c + 1], noff = q1 - q0;
        auto tile = [&](int s) { return s >= noff ? a.diag[c] : FWD ? a.row_tiles[q0 + s] : a.col_tiles[q1 - 1 - s]; };
        dd_t v = dd_zero(); // thread t < 64: entry t
        if (tid < nb) v = ld_dd(a.x + r0 + tid);
        int t = tile(0);
        sp_load_tile(sp_sm, a.tiles + (long)t * SP_T * SP_T, tid, SP_THREADS);
        if (tid < SP_T) msk[0][tid] = a.mask[(long)t * SP_T + tid];
        for (int s = 0; s < noff; ++s) {
            const int buf = s & 1, p = a.tIJ[2 * t + (FWD ? 1 : 0)], tn = tile(s + 1);
            double2 *T = sp_sm + buf * SP_T * SPL;
            if (warp < 2) {
                if (!sp_wait(a, p)) {
                    if (lane == 0) fail = 1;
                } else if (p * SP_T + tid < a.m) {
                    const dd_t xa = sp_ldcg(a.x + p * SP_T + tid);
                    xs[tid] = make_double2(xa.hi, xa.lo);
                }
            }
            __syncthreads(); // the tile and block p are in
            if (fail) return;
            for (int e = tid; e < SP_T * SP_T; e += SP_THREADS) {
                const int i = e & (SP_T - 1), j = e >> 6;
                if (!bit64(msk[buf][j], i)) continue;
                const double2 xt = xs[FWD ? j : i];
                sm_st(T, i, j, dd_mul(sm_dd(T, i, j), dd_make(xt.x, xt.y)));
            }
            __syncthreads(); // its products are formed
            if (warp >= 2) {
                sp_load_tile(sp_sm + (buf ^ 1) * SP_T * SPL, a.tiles + (long)tn * SP_T * SP_T, tid - 64, SP_THREADS - 64);
                if (tid >= 64 && tid < 64 + SP_T) msk[buf ^ 1][tid - 64] = a.mask[(long)tn * SP_T + tid - 64];
            } else {
                // the steps in which some entry of this warp takes a term
                unsigned lo, hi;
                bool full; // every entry of the warp takes all 64
                if (FWD) {
                    const unsigned a0 = (unsigned)(msk[buf][lane] >> (32 * warp)), a1 = (unsigned)(msk[buf][32 + lane] >> (32 * warp));
                    lo = __ballot_sync(0xffffffffu, a0 != 0u);
                    hi = __ballot_sync(0xffffffffu, a1 != 0u);
                    full = __all_sync(0xffffffffu, (a0 & a1) == 0xffffffffu);
                } else {
                    const unsigned a0 = (unsigned)msk[buf][tid], a1 = (unsigned)(msk[buf][tid] >> 32);
                    lo = __reduce_or_sync(0xffffffffu, a0);
                    hi = __reduce_or_sync(0xffffffffu, a1);
                    full = __all_sync(0xffffffffu, (a0 & a1) == 0xffffffffu);
                }
                auto product = [&](int q) { return FWD ? T[tid + SPL * q] : T[q + SPL * tid]; };
                auto takes = [&](int q) { return FWD ? bit64(msk[buf][q], tid) : bit64(msk[buf][tid], q); };
                if (full) {
                    double2 z[2][8]; // the next eight products come while these are subtracted
#pragma unroll
                    for (int u = 0; u < 8; ++u) z[0][u] = product(FWD ? u : 63 - u);
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (g < 7) z[(g + 1) & 1][u] = product(FWD ? 8 * g + 8 + u : 55 - 8 * g - u);
#pragma unroll
                        for (int u = 0; u < 8; ++u) v = dd_sub(v, dd_make(z[g & 1][u].x, z[g & 1][u].y));
                    }
                    lo = hi = 0u;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int base = (FWD ? h : 1 - h) * 32;
                    unsigned left = base ? hi : lo;
                    if (left == 0u) continue;
                    auto next = [&] {
                        const int q = FWD ? __ffs(left) - 1 : 31 - __clz(left);
                        left &= ~(1u << q);
                        return base + q;
                    };
                    int q = next();
                    double2 z = product(q);
                    bool b = takes(q);
                    while (left != 0u) {
                        q = next();
                        const double2 zn = product(q);
                        const bool bn = takes(q);
                        const dd_t u = dd_sub(v, dd_make(z.x, z.y));
                        v = b ? u : v;
                        z = zn;
                        b = bn;
                    }
                    const dd_t u = dd_sub(v, dd_make(z.x, z.y));
                    v = b ? u : v;
                }
            }
            t = tn;
        }
        if (tid < SP_T) vs[tid] = make_double2(v.hi, v.lo);
        __syncthreads(); // the diagonal tile is in
        if (warp == 0) {
            dd_t v0 = dd_make(vs[lane].x, vs[lane].y), v1 = dd_make(vs[32 + lane].x, vs[32 + lane].y);
            sp_diag<FWD>(sp_sm + (noff & 1) * SP_T * SPL, msk[noff & 1], nb, v0, v1);
            if (r0 + lane < a.m) st_dd(a.x + r0 + lane, v0);
            if (r0 + 32 + lane < a.m) st_dd(a.x + r0 + 32 + lane, v1);
            __threadfence();
            __syncwarp();
            if (lane == 0 && c != a.withhold) sp_st_release(a.flags + c, a.epoch);
        }
        __syncthreads();
    }
}

__global__ void sp_permute_kernel(const dd_t *x, const int *order, int m, dd_t *xp) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) st_dd(xp + k, ld_dd(x + order[k]));
}
__global__ void sp_unpermute_kernel(const dd_t *xp, const int *order, int m, dd_t *x) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) st_dd(x + order[k], ld_dd(xp + k));
}

// ============================================================== host side
static void upload_schedule(Context &c, SparseDev &s) {
    const TileSchedule &t = s.sched;
    cudaStream_t st = c.stream;
    std::vector<int> tij(2 * (size_t)t.ntiles), diag(t.nblk);
    for (int k = 0; k < t.ntiles; ++k) {
        tij[2 * k] = t.tI[k];
        tij[2 * k + 1] = t.tJ[k];
    }
    for (int J = 0; J < t.nblk; ++J) diag[J] = t.tile_of[J + (size_t)t.nblk * J];
    s.tIJ.upload(tij, st);
    s.diag.upload(diag, st);
    s.tile_of.upload(t.tile_of, st);
    std::vector<unsigned long long> mk(t.mask.begin(), t.mask.end());
    s.mask.upload(mk, st);
    s.col_ptr.upload(t.col_ptr, st);
    s.col_tiles.upload(t.col_tiles.empty() ? std::vector<int>{0} : t.col_tiles, st);
    s.row_ptr.upload(t.row_ptr, st);
    s.row_tiles.upload(t.row_tiles.empty() ? std::vector<int>{0} : t.row_tiles, st);
    s.upd.upload(t.upd.empty() ? std::vector<int>{0} : t.upd, st);
    s.tiles.alloc((size_t)t.ntiles * SP_T * SP_T);
    s.xp.alloc(std::max(1, t.m));
    s.panel_done.alloc(std::max(1, t.nblk));
    CK(cudaMemsetAsync(s.panel_done.p, 0, sizeof(int) * std::max(1, t.nblk), st));
    s.drop_graph();
    // per entry of the reference layout: its column b and row a
    const SparseStructure &ss = s.plan.s;
    std::vector<int> eb(ss.nnz()), ea(ss.nnz());
    for (int b = 0; b < ss.m; ++b)
        for (int q = ss.rowptr[b]; q < ss.rowptr[b + 1]; ++q) {
            eb[q] = b;
            ea[q] = ss.col[q];
        }
    s.ent_b.upload(eb, st);
    s.ent_a.upload(ea, st);
    CK(cudaStreamSynchronize(st));
}

void sparse_setup(Context &c) {
    if (!c.sp) c.sp = new SparseDev();
    SparseDev &s = *c.sp;
    s.plan = plan_schur(c.prob, c.schur_mode);
    s.active = s.plan.sparse;
    if (!s.active) return;
    s.sched = make_tile_schedule(s.plan.s);
    s.order.upload(s.plan.order, c.stream);
    upload_schedule(c, s);
}

void sparse_setup_structure(Context &c, const SparseStructure &ss) {
    const std::string bad = check_structure(ss);
    if (!bad.empty()) throw Error(ERR_ARG, "sparse factor structure: " + bad);
    if (!c.sp) c.sp = new SparseDev();
    SparseDev &s = *c.sp;
    s.plan = SparsePlan();
    s.plan.sparse = true;
    s.plan.s = ss;
    s.plan.order.resize(ss.m);
    for (int i = 0; i < ss.m; ++i) s.plan.order[i] = i;
    s.plan.extended = 2 * ss.nnz() - ss.m;
    s.active = true;
    s.sched = make_tile_schedule(ss);
    s.order.upload(s.plan.order, c.stream);
    upload_schedule(c, s);
}

// The launches of one factorisation.  Panel J waits for every update that
// writes into its column block; the update of panel J waits for panel J and
// for the previous update of each tile it writes (updates of one tile stay
// in pivot order).  Panels of independent subtrees of the elimination run
// side by side.
static void sparse_launches(Context &c, cudaGraph_t g) {
    SparseDev &s = *c.sp;
    const TileSchedule &t = s.sched;
    CK(cudaFuncSetAttribute(sp_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SP_PANEL_SMEM));
    CK(cudaFuncSetAttribute(sp_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SP_TWO_TILES));
    std::vector<cudaGraphNode_t> last_writer(t.ntiles, nullptr);
    std::vector<std::vector<cudaGraphNode_t>> into(t.nblk);
    auto uniq = [](std::vector<cudaGraphNode_t> v) {
        std::sort(v.begin(), v.end());
        v.erase(std::unique(v.begin(), v.end()), v.end());
        return v;
    };
    dd_t *tiles = s.tiles.p;
    const unsigned long long *mask = s.mask.p;
    int m = t.m;
    int *done = s.panel_done.p;
    for (int J = 0; J < t.nblk; ++J) {
        const int ncol = t.col_ptr[J + 1] - t.col_ptr[J];
        int diag = t.tile_of[J + (size_t)t.nblk * J];
        const size_t smem = ncol > 0 ? SP_PANEL_SMEM : SP_TILE_SMEM;
        const int *col = s.col_tiles.p + t.col_ptr[J];
        int Jv = J;
        cudaGraphNode_t pnode = nullptr;
        {
            void *args[] = {&tiles, &mask, &m, &Jv, &diag, &col, &done};
            cudaKernelNodeParams kp{};
            kp.func = (void *)sp_panel_kernel;
            kp.gridDim = dim3(1 + 2 * ncol);
            kp.blockDim = dim3(SP_PANEL_THREADS);
            kp.sharedMemBytes = (unsigned)smem;
            kp.kernelParams = args;
            const std::vector<cudaGraphNode_t> deps = uniq(into[J]);
            CK(cudaGraphAddKernelNode(&pnode, g, deps.data(), deps.size(), &kp));
        }
        // the update of panel J in two nodes: the targets in column block
        // J + 1 (listed first: the schedule sorts targets by column block),
        // which panel J + 1 waits for, and the rest, which run beside it
        int nbJ = std::min(SP_T, t.m - J * SP_T);
        const int q0 = t.upd_ptr[J], q1 = t.upd_ptr[J + 1];
        int qs = q0;
        while (qs < q1 && t.tJ[t.upd[3 * qs]] == J + 1) ++qs;
        for (int part = 0; part < 2; ++part) {
            const int a = part == 0 ? q0 : qs, b = part == 0 ? qs : q1;
            if (a == b) continue;
            const int *upd = s.upd.p + 3 * (size_t)a;
            void *args[] = {&tiles, &mask, &upd, &nbJ};
            cudaKernelNodeParams kp{};
            kp.func = (void *)sp_update_kernel;
            kp.gridDim = dim3((b - a) * SP_UPD_SPLIT);
            kp.blockDim = dim3(SP_THREADS);
            kp.sharedMemBytes = (unsigned)SP_TWO_TILES;
            kp.kernelParams = args;
            std::vector<cudaGraphNode_t> deps{pnode};
            for (int q = a; q < b; ++q)
                if (last_writer[t.upd[3 * q]]) deps.push_back(last_writer[t.upd[3 * q]]);
            deps = uniq(deps);
            cudaGraphNode_t unode;
            CK(cudaGraphAddKernelNode(&unode, g, deps.data(), deps.size(), &kp));
            for (int q = a; q < b; ++q) {
                const int target = t.upd[3 * q];
                last_writer[target] = unode;
                into[t.tJ[target]].push_back(unode);
            }
        }
    }
}

static void sparse_panels(Context &c) {
    SparseDev &s = *c.sp;
    if (!s.graph) {
        cudaGraph_t g;
        CK(cudaGraphCreate(&g, 0));
        try {
            sparse_launches(c, g);
            CK(cudaGraphInstantiate(&s.graph, g, 0));
        } catch (...) {
            cudaGraphDestroy(g);
            throw;
        }
        CK(cudaGraphDestroy(g));
    }
    CK(cudaGraphLaunch(s.graph, c.stream));
}

void sparse_factor_B(Context &c) {
    SparseDev &s = *c.sp;
    PROF_SCOPE("sparse_factor", c.stream);
    if (s.sched.ntiles == 0) return;
    sp_gather_B_kernel<<<s.sched.ntiles, SP_THREADS, 0, c.stream>>>(c.B.p, c.m, s.order.p, s.tIJ.p, s.mask.p, s.tiles.p);
    CK_LAUNCH();
    sparse_panels(c);
}

void sparse_load_values(Context &c, const dd_t *vals) {
    SparseDev &s = *c.sp;
    const long nnz = s.plan.s.nnz();
    if (s.sched.ntiles == 0) return;
    CK(cudaMemsetAsync(s.tiles.p, 0, sizeof(dd_t) * (size_t)s.sched.ntiles * SP_T * SP_T, c.stream));
    sp_scatter_kernel<<<ceil_div(nnz, 256), 256, 0, c.stream>>>(vals, s.ent_b.p, s.ent_a.p, nnz, s.tile_of.p, s.sched.nblk, s.tiles.p);
    CK_LAUNCH();
}

void sparse_factor_values(Context &c, const dd_t *vals) {
    PROF_SCOPE("sparse_factor", c.stream);
    sparse_load_values(c, vals);
    if (c.sp->sched.ntiles > 0) sparse_panels(c);
}

void sparse_values(Context &c, dd_t *vals) {
    SparseDev &s = *c.sp;
    const long nnz = s.plan.s.nnz();
    if (nnz == 0) return;
    sp_gather_kernel<<<ceil_div(nnz, 256), 256, 0, c.stream>>>(s.tiles.p, s.ent_b.p, s.ent_a.p, nnz, s.tile_of.p, s.sched.nblk, vals);
    CK_LAUNCH();
}

static int sp_grid_cap(const void *kernel) {
    int dev = 0, sms = 0, per = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SP_SOLVE_SMEM));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, SP_THREADS, SP_SOLVE_SMEM));
    if (per < 1) throw Error(ERR_CUDA, "sparse solve: the wave kernel does not fit on an SM");
    return per * sms;
}

static void sp_solve_dir(Context &c, char dir, dd_t *x) {
    SparseDev &s = *c.sp;
    const TileSchedule &t = s.sched;
    TrsvSync &sync = trsv_sync(c, t.m);
    if (++sync.epoch <= 0) sync.epoch = 1;
    SpSolveArgs a{s.tiles.p, s.mask.p, s.tIJ.p, s.row_ptr.p, s.row_tiles.p, s.col_ptr.p, s.col_tiles.p, s.diag.p, t.m, t.nblk, sync.epoch, x,
                  sync.flags, sync.flags + sync.capacity, sync.wait_ns, sync.withhold};
    const void *k = dir == 'N' ? (const void *)sp_solve_kernel<true> : (const void *)sp_solve_kernel<false>;
    static thread_local int cap[2][64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int &cp = cap[dir == 'N' ? 0 : 1][dev & 63];
    if (cp == 0) cp = sp_grid_cap(k);
    const int grid = std::min(t.nblk, cp);
    void *args[] = {&a};
    CK(cudaLaunchCooperativeKernel(k, grid, SP_THREADS, args, SP_SOLVE_SMEM, c.stream));
    CK_LAUNCH();
}

void sparse_solve_raw(Context &c, dd_t *x) {
    if (c.sp->sched.m == 0) return;
    PROF_SCOPE("sparse_solve", c.stream);
    sp_solve_dir(c, 'N', x);
    sp_solve_dir(c, 'T', x);
    trsv_check(c.stream, c.trsv);
}

void sparse_solve(Context &c, dd_t *x) {
    SparseDev &s = *c.sp;
    const int m = s.sched.m;
    if (m == 0) return;
    PROF_SCOPE("sparse_solve", c.stream);
    sp_permute_kernel<<<ceil_div(m, 256), 256, 0, c.stream>>>(x, s.order.p, m, s.xp.p);
    CK_LAUNCH();
    sp_solve_dir(c, 'N', s.xp.p);
    sp_solve_dir(c, 'T', s.xp.p);
    sp_unpermute_kernel<<<ceil_div(m, 256), 256, 0, c.stream>>>(s.xp.p, s.order.p, m, x);
    CK_LAUNCH();
    trsv_check(c.stream, c.trsv);
}

double sparse_chol_terms(const Context &c) { return c.sp ? (double)c.sp->sched.exact_terms : 0.0; }

} // namespace sddd
