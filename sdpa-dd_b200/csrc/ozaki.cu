// Tensor-core split of the Cholesky trailing update, C(lower) -= P P^T.
//
// Split (ozaki_split_kernel).  Row r of the panel is scaled by 2^-e_r, with
// e_r chosen so that every |P(r,k)| 2^-e_r <= 0.498, and written as a fixed
// point number in B signed base-256 digits D_1 .. D_B in [-128, 127]:
//   P(r,k) = 2^e_r sum_s D_s(r,k) 2^-8s  (+ remainder <= 2^-(8B+1) 2^e_r).
// 0.498 < 127/255, the largest value that digits up to 127 reach, so a row whose
// largest entry lies in the top 0.4 % below a power of two takes a scale one bit
// larger than 7-bit digits (in [-64, 64]) need.  A caller's S 7-bit slices are
// therefore carried by B = ceil((7S + 1)/8) digits, so that every row keeps the
// 7S bits below its largest entry (16 slices: 15 digits, truncated at 2^-120;
// 120 digit products replace 136).  With 14 digits the error of such rows'
// products was 3.6 times that of 16 7-bit digits (rms, small entries beside the
// largest one: 2^-107.0 of the power of two against 2^-108.8); with 15 it is
// 2^-113.9, at 5 % of the update's time.
//
// Products (ozaki_syrk_kernel).  C(i,j) -= 2^(e_i+e_j) sum_d 2^-8d A_d(i,j),
// A_d = sum_{s+t=d} D_s(i,:) . D_t(j,:), for d = 2..B+1 (the B(B+1)/2 digit
// pairs that reach 8(B+1) bits).  Every A_d is an exact int32 (|A_d| <=
// (d-1) * 64 * 128 * 128 < 2^24, d <= 16), accumulated by tcgen05.mma kind::i8 in
// tensor memory.
//
// One tcgen05.mma costs about the same time for any N up to 128 (on B200 a
// kind::i8 M=128 K=32 instruction occupies the issuing thread ~97 cycles
// for N = 32..128 and ~170 for N = 256), so the kernel issues few, wide
// MMAs: a tile is 128 rows x 16 columns, its B operand the tile's digits
// stacked (row 16 (t-1) + j is digit t of column j), and its accumulators
// are laid out by diagonal (diagonal d in columns 16 (d-2) .. 16 (d-2) + 15).
// The MMA of A digit s against stacked B digits 1 .. B+1-s (N = 16 (B+1-s))
// then writes diagonals s+1 .. B+1 in one instruction: B x 2 K steps = 30
// MMAs per tile for 15 digits.
//
// Epilogue: an entry's diagonals combine exactly to four 64-bit integers
// (oz_groups), which become doubles scaled by 2^(e_i+e_j) and are summed with
// C's two halves (oz_sub).
//
// Kernel layout: one persistent CTA per SM over the tiles of the lower
// triangle (row-block major, so a CTA keeps its 128-row A digits in shared
// memory while it walks the columns).  Bulk copies (cp.async.bulk, no multicast)
// stage everything: warp 17 the digits, B two tiles deep, and warp 18 C's tiles,
// two deep, a copy per column (clipped to the lower triangle).  Warp 0 lane 0
// issues the MMAs; warps 1-16 drain tensor memory, which holds two
// accumulator buffers, so one tile multiplies while the last drains.
// Operand layout in global memory: 16-row blocks, in a block digit by digit,
// a digit's 16 rows as two 8-row groups of 512 bytes, each four 128-byte core
// matrices (8 rows x 16 K-bytes): the K-major, non-swizzled canonical layout
// of the MMA's shared-memory descriptors (LBO 128 bytes between the two K
// chunks of one MMA, SBO 512 bytes between row groups), so a tile's stacked B
// digits are one copy; the A digits of a row block are gathered digit by
// digit, 1 KB at a time.
// Every mbarrier wait is bounded (the context's wait budget, 2 s by
// default); on expiry the CTA records a code in
// the error word, stops issuing, waits (bounded) for what it issued and
// frees its tensor memory.
//
// What bounds it: C is read and written once per panel (32 bytes an entry of
// the lower triangle, 0.24 ms at n = 9920) and a tile's 30 MMAs take about as
// long, but FP64 and tensor instructions wait for one another (see the
// epilogue), so a tile takes the sum of the two.  Measured, one update: n =
// 9920 476 us, n = 5000 141, n = 2000 35; with 14 digits 454, 134 and 33.5; with
// 16 7-bit digits assembled in FP64, C loaded by the epilogue's threads and the
// copies issued by the MMA's thread 529, 154 and 33.
#include "ozaki.h"

#include <algorithm>
#include <string>

#include "bulk.cuh"
#include "prof.h"

namespace sddd {

namespace {

constexpr int OZ_EPI_WARPS = 16; // epilogue warps: four per tensor-memory lane quadrant
constexpr int OZ_EPI_COLS = OZ_COLS_B / (OZ_EPI_WARPS / 4); // tile columns per epilogue thread
constexpr int OZ_AB_WARP = 1 + OZ_EPI_WARPS, OZ_C_WARP = 2 + OZ_EPI_WARPS; // the warps that copy the operands and C
constexpr int OZ_THREADS = 32 * (3 + OZ_EPI_WARPS); // warp 0: MMA; then the epilogue; then the copies
// 19 warps put five on an SM sub-partition: 5 x 32 x 96 registers fit its 16384
constexpr int OZ_MAX_REGS = 96;
constexpr int OZ_A_BYTES = OZ_ROWS_A * OZ_K; // one digit of a 128-row block
constexpr int OZ_B_BYTES = OZ_COLS_B * OZ_K; // one digit of a 16-row block
constexpr int OZ_TILE_B = OZ_MAX_DIGITS * OZ_B_BYTES; // the stacked B digits of a tile
constexpr int OZ_STAGES = 2;                 // B tiles in shared memory
constexpr int OZ_C_STAGES = 2;               // C tiles in shared memory
constexpr int OZ_C_BYTES = OZ_ROWS_A * OZ_COLS_B * 16; // one C tile
constexpr int OZ_ACC_COLS = 256; // tensor-memory columns of one accumulator buffer
static_assert(2 * OZ_ACC_COLS <= 512, "split kernel: two accumulator buffers must fit tensor memory");
static_assert(OZ_MAX_DIGITS * OZ_COLS_B <= OZ_ACC_COLS, "split kernel: the widest MMA has N = 16 B <= 256");
// the A digits of a row block, OZ_STAGES stacked B tiles and OZ_C_STAGES C tiles
constexpr size_t OZ_SMEM = 1024 + (size_t)OZ_MAX_DIGITS * OZ_A_BYTES + (size_t)OZ_STAGES * OZ_TILE_B + (size_t)OZ_C_STAGES * OZ_C_BYTES;
static_assert(OZ_SMEM <= 232448 - 512, "split kernel: shared memory above the per-CTA limit");
// kind::i8 instruction descriptor: D s32, A and B s8, both K-major, M = 128,
// N = n (a multiple of 16, 16..256).
__host__ __device__ constexpr uint32_t oz_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZ_ROWS_A >> 4) << 24);
}

__device__ __forceinline__ unsigned long long oz_ns() { return globaltimer_ns(); }
// Waits for the phase with the given parity to complete; false when the CTA
// is aborting or the wait ran out (then the CTA aborts with `code`).
__device__ bool oz_wait(uint64_t *b, uint32_t parity, volatile int *abort_flag, int *err, int code, unsigned long long wait_ns) {
    // the clock is read only once a wait has become long
    for (int k = 0; k < 64; ++k)
        if (mbar_try_wait(b, parity)) return true;
    const unsigned long long t0 = oz_ns();
    while (!mbar_try_wait(b, parity)) {
        if (*abort_flag) return false;
        if (oz_ns() - t0 > wait_ns) {
            *abort_flag = 1;
            atomicCAS(err, 0, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, no swizzle, LBO 128, SBO 512,
// descriptor version 1.
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46);
}

struct OzArgs {
    const int8_t *digits; // by 16-row block, a block's nd digits back to back
    const int *exps;
    dd_t *C;
    long ldc;
    int n, nd, nI, nJ;
    int skip; // rows below skip are not written (their block is updated elsewhere)
    long tiles;
    int *err;
    unsigned long long wait_ns; // budget of one mbarrier wait
};

// Tiles of the lower triangle, row-block major: row block I (128 rows) has
// min(8 (I + 1), nJ) column blocks of 16.
constexpr int OZ_JPI = OZ_ROWS_A / OZ_COLS_B;
__device__ __forceinline__ void oz_tile_at(long t, int nI, int nJ, int &I, int &J) {
    I = 0;
    for (; I < nI; ++I) {
        const long cnt = min((long)OZ_JPI * (I + 1), (long)nJ);
        if (t < cnt) break;
        t -= cnt;
    }
    J = (int)t;
}
__device__ __forceinline__ void oz_tile_next(int nJ, int &I, int &J) {
    if (++J >= min(OZ_JPI * (I + 1), nJ)) {
        ++I;
        J = 0;
    }
}

// Shared state of one CTA.
//   barA          A digits of the current row block landed
//   barB[st]      the B digits of the tile in stage st landed
//   done[st]      every MMA of the tile in stage st completed: its
//                 accumulators are there, and the stage (at a row-block
//                 change A as well) may be reloaded
//   tempty[b]     accumulator buffer b is drained
//   cfull/cempty  C stage st holds its tile's entries / has been read
//   fin           every MMA the CTA issued completed (exit)
struct OzShared {
    uint64_t barA, barB[OZ_STAGES], done[OZ_STAGES], tempty[2], cfull[OZ_C_STAGES], cempty[OZ_C_STAGES], fin;
    uint32_t tmem;
    int abort_flag;
};

__device__ __forceinline__ void tc_mma_i8_n(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(da),
                 "l"(db), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// MMAs of one tile into the accumulator buffer at dbuf, A digits S0 .. S1:
// for A digit s and K step kk, one MMA against the stacked B digits t = 1 ..
// B+1-s (N = 16 (B+1-s)) writes the columns of diagonals s+1 .. B+1.  The
// first (s = 1, N = 16 B) covers every column and overwrites; the rest
// accumulate.
template <int ND, int S0, int S1>
__device__ __forceinline__ void oz_issue(uint32_t dbuf, uint64_t descA, uint64_t descB) {
#pragma unroll
    for (int s = S0; s <= S1; ++s) {
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)
            tc_mma_i8_n(dbuf + (uint32_t)((s - 1) * OZ_COLS_B), descA + (uint64_t)(((s - 1) * OZ_A_BYTES + kk * 256) >> 4),
                        descB + (uint64_t)((kk * 256) >> 4), oz_idesc((ND + 1 - s) * OZ_COLS_B), (s == 1 && kk == 0) ? 0u : 1u);
    }
}
__device__ __forceinline__ void oz_issue_rt(int nd, int s0, int s1, uint32_t dbuf, uint64_t descA, uint64_t descB) {
    for (int s = s0; s <= s1; ++s)
        for (int kk = 0; kk < 2; ++kk)
            tc_mma_i8_n(dbuf + (uint32_t)((s - 1) * OZ_COLS_B), descA + (uint64_t)(((s - 1) * OZ_A_BYTES + kk * 256) >> 4),
                        descB + (uint64_t)((kk * 256) >> 4), oz_idesc((nd + 1 - s) * OZ_COLS_B), (s == 1 && kk == 0) ? 0u : 1u);
}

// A wait that ignores the abort flag (still bounded): used on the way out,
// where copies and MMAs already issued must finish before the CTA releases
// its shared and tensor memory.
__device__ void oz_wait_out(uint64_t *b, uint32_t parity, int *err, unsigned long long wait_ns) {
    const unsigned long long t0 = oz_ns();
    while (!mbar_try_wait(b, parity)) {
        if (oz_ns() - t0 > wait_ns) {
            atomicCAS(err, 0, 5);
            return;
        }
    }
}

// Warp 0, lane 0: the MMAs (tile n from B stage n mod OZ_STAGES into
// accumulator buffer n mod 2).  It only waits and issues: an MMA holds the
// issuing thread for about its own duration, so whatever else this thread
// does the tensor pipe stands idle for.  The next tile's barriers (a try
// costs over 100 cycles even when it succeeds) are tried before the last
// MMAs of a tile are issued.
__device__ void oz_mma(const OzArgs &a, OzShared &S, const uint8_t *smA, const uint8_t *smB, int I, int J, int ntile) {
    volatile int *abort_flag = &S.abort_flag;
    const uint64_t descA = oz_desc(smem_u32(smA));
    const uint64_t descB0 = oz_desc(smem_u32(smB));
    uint32_t phA = 0, phB = 0;
    int st = 0, curA = -1, n = 0;
    bool haveB = false, haveT = false; // tile n's B digits are there, its buffer is drained
    for (; n < ntile; ++n) {
        const int b = n & 1;
        if (I != curA) {
            if (!oz_wait(&S.barA, phA, abort_flag, a.err, 2, a.wait_ns)) break;
            phA ^= 1u;
            curA = I;
        }
        if (!haveB && !oz_wait(&S.barB[st], phB, abort_flag, a.err, 3, a.wait_ns)) break;
        if (!haveT && !oz_wait(&S.tempty[b], (uint32_t)(((n >> 1) & 1) ^ 1), abort_flag, a.err, 4, a.wait_ns)) break;
        tc_fence_after();
        const uint64_t descB = descB0 + (uint64_t)((st * OZ_TILE_B) >> 4);
        const uint32_t dbuf = S.tmem + (uint32_t)(b * OZ_ACC_COLS);
        constexpr int HEAD = OZ_MAX_DIGITS - 2;
        const bool full = a.nd == OZ_MAX_DIGITS;
        if (full)
            oz_issue<OZ_MAX_DIGITS, 1, HEAD>(dbuf, descA, descB);
        else
            oz_issue_rt(a.nd, 1, a.nd, dbuf, descA, descB);
        const int stn = st + 1 == OZ_STAGES ? 0 : st + 1;
        const uint32_t phn = stn == 0 ? phB ^ 1u : phB;
        haveB = n + 1 < ntile && mbar_try_wait(&S.barB[stn], phn);
        haveT = n + 1 < ntile && mbar_try_wait(&S.tempty[b ^ 1], (uint32_t)((((n + 1) >> 1) & 1) ^ 1));
        if (full) oz_issue<OZ_MAX_DIGITS, HEAD + 1, OZ_MAX_DIGITS>(dbuf, descA, descB);
        tc_commit(&S.done[st]);
        st = stn;
        phB = phn;
        oz_tile_next(a.nJ, I, J);
    }
    // every issued MMA completes (bounded wait) before the CTA frees its memory
    if (n > 0) {
        tc_commit(&S.fin);
        oz_wait_out(&S.fin, 0, a.err, a.wait_ns);
    }
}

// Lane 0 waits, the warp follows its outcome.
__device__ __forceinline__ bool oz_wait_lane0(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *err, int code, unsigned long long wait_ns) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = oz_wait(bar, parity, abort_flag, err, code, wait_ns) ? 1 : 0;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Warp OZ_AB_WARP: the operands.  B's digits OZ_STAGES tiles deep, one copy a
// tile; the A digits of a row block when it changes, once the MMAs of the tile
// before have read the old ones, 1 KB a copy over all lanes.
__device__ void oz_load_ab(const OzArgs &a, OzShared &S, uint8_t *smA, uint8_t *smB, int I, int J, int ntile) {
    volatile int *abort_flag = &S.abort_flag;
    const int lane = threadIdx.x & 31, nd = a.nd;
    int curA = -1, nA = 0, nB = 0; // copies issued
    int st = 0, last = 0;          // B stage of this tile and of the one before
    uint32_t ph = 0, phlast = 0;   // parity of the stage's current use
    for (int n = 0; n < ntile; ++n) {
        if (n >= OZ_STAGES && !oz_wait_lane0(&S.done[st], ph ^ 1u, abort_flag, a.err, 1, a.wait_ns)) break;
        if (lane == 0) {
            mbar_expect_tx(&S.barB[st], (uint32_t)(nd * OZ_B_BYTES));
            bulk_g2s(smB + (size_t)st * OZ_TILE_B, a.digits + (long)J * nd * OZ_B_BYTES, (uint32_t)(nd * OZ_B_BYTES), &S.barB[st]);
        }
        nB = n + 1;
        if (I != curA) {
            if (n > 0 && !oz_wait_lane0(&S.done[last], phlast, abort_flag, a.err, 1, a.wait_ns)) break;
            if (lane == 0) mbar_expect_tx(&S.barA, (uint32_t)(nd * OZ_A_BYTES));
            __syncwarp();
            const int8_t *src = a.digits + (long)I * OZ_JPI * nd * OZ_B_BYTES;
            for (int e = lane; e < nd * OZ_JPI; e += 32) { // 16-row block q, digit s
                const int s = e / OZ_JPI, q = e % OZ_JPI;
                bulk_g2s(smA + (size_t)s * OZ_A_BYTES + q * OZ_B_BYTES, src + (long)(q * nd + s) * OZ_B_BYTES, OZ_B_BYTES, &S.barA);
            }
            ++nA;
            curA = I;
        }
        last = st;
        phlast = ph;
        if (++st == OZ_STAGES) {
            st = 0;
            ph ^= 1u;
        }
        oz_tile_next(a.nJ, I, J);
    }
    // every issued copy lands (bounded waits) before the CTA leaves
    if (lane == 0) {
        if (nA > 0) oz_wait_out(&S.barA, (uint32_t)((nA - 1) & 1), a.err, a.wait_ns);
        for (int k = max(0, nB - OZ_STAGES); k < nB; ++k) oz_wait_out(&S.barB[k % OZ_STAGES], (uint32_t)((k / OZ_STAGES) & 1), a.err, a.wait_ns);
    }
    __syncwarp();
}

// Warp OZ_C_WARP: C's tiles OZ_C_STAGES deep; lane c copies column c's rows
// of the lower triangle (16-byte entries, so any row is a valid start).
__device__ void oz_load_c(const OzArgs &a, OzShared &S, uint8_t *smC, int I, int J, int ntile) {
    volatile int *abort_flag = &S.abort_flag;
    const int lane = threadIdx.x & 31;
    int nC = 0; // tiles whose copies are issued
    for (; nC < ntile; ++nC) {
        const int cs = nC % OZ_C_STAGES;
        if (!oz_wait_lane0(&S.cempty[cs], (uint32_t)(((nC / OZ_C_STAGES) & 1) ^ 1), abort_flag, a.err, 7, a.wait_ns)) break;
        const int j = J * OZ_COLS_B + lane;
        int bytes = 0, r0 = 0;
        if (lane < OZ_COLS_B && j < a.n) {
            r0 = max(I * OZ_ROWS_A, max(j, a.skip));
            bytes = max(0, min(I * OZ_ROWS_A + OZ_ROWS_A, a.n) - r0) * 16;
        }
        const int total = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_expect_tx(&S.cfull[cs], (uint32_t)total);
        __syncwarp();
        if (bytes > 0)
            bulk_g2s(smC + (size_t)cs * OZ_C_BYTES + (size_t)lane * (OZ_ROWS_A * 16) + (size_t)(r0 - I * OZ_ROWS_A) * 16, a.C + r0 + a.ldc * (long)j,
                     (uint32_t)bytes, &S.cfull[cs]);
        oz_tile_next(a.nJ, I, J);
    }
    // every issued copy lands (bounded waits) before the CTA leaves
    if (lane == 0)
        for (int k = max(0, nC - OZ_C_STAGES); k < nC; ++k) oz_wait_out(&S.cfull[k % OZ_C_STAGES], (uint32_t)((k / OZ_C_STAGES) & 1), a.err, a.wait_ns);
    __syncwarp();
}

__device__ __forceinline__ void tc_ld2(uint32_t taddr, int32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}

// The diagonals of one entry, v[0..14] (diagonal d at v[d-2]; those beyond
// B+1 are zero), as four exact integers in units of 2^-40, 2^-72, 2^-104 and
// 2^-136: A_2..A_5, A_6..A_9, A_10..A_13, A_14..A_16.  |A_d| <= (d-1) 2^20, so
// each is below 2^49.
__device__ __forceinline__ void oz_groups(const int32_t (*v)[2], int c, long long *w) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
        w[j] = (((long long)v[4 * j][c] * 16777216 + (long long)v[4 * j + 1][c] * 65536) + (long long)v[4 * j + 2][c] * 256) + v[4 * j + 3][c];
    w[3] = ((long long)v[12][c] * 16777216 + (long long)v[13][c] * 65536) + (long long)v[14][c] * 256;
}

// The group w 2^e as a double: the bits of (2^52 + 2^51 + w) 2^e, then one
// exact subtraction; k holds the upper word of (2^52 + 2^51) 2^e.
__device__ __forceinline__ double oz_scaled(long long w, int k) {
    return __hiloint2double((int)(w >> 32) + k, (int)w) - __hiloint2double(k, 0);
}

// C - (g0 + g1 + g2 + g3) as a dd, the groups already scaled.  The two
// leading pairs are summed without error; what is rounded is the sum of their
// errors and of the two small groups (below 2^-56 of 2^(e_i+e_j): 2^-109 of
// it at most) and the result's own low part (2^-105 of the result).
__device__ __forceinline__ dd_t oz_sub(double2 c, double g0, double g1, double g2, double g3) {
    double e, f, g, l, lo;
    const double s = ddm::two_sum(c.x, -g0, e);
    const double t = ddm::two_sum(c.y, -g1, f);
    const double u = ddm::two_sum(e, t, g);
    const double r = (f + g) - (g2 + g3);
    const double h = ddm::two_sum(s, u, l);
    const double hi = ddm::fast_two_sum(h, l + r, lo);
    return dd_make(hi, lo);
}

// The diagonals of columns col and col + 1 of a thread's row; nd of them.
__device__ __forceinline__ void oz_drain2(uint32_t taddr, int nd, int32_t (*v)[2]) {
#pragma unroll
    for (int u = 0; u < OZ_MAX_DIGITS; ++u) {
        if (u < nd) {
            tc_ld2(taddr + (uint32_t)(u * OZ_COLS_B), v[u]);
        } else {
            v[u][0] = 0;
            v[u][1] = 0;
        }
    }
    tc_wait_ld();
}

// One thread's entries of a tile in which the warp meets scales at the ends of
// the exponent range: the groups scaled one by one (out of line, so that the
// common case keeps its registers).
__device__ __noinline__ void oz_tile_far(uint32_t taddr, int nd, const double2 *ct, dd_t *cp, long ldc, int ncol, int ei, const int *ej) {
#pragma unroll 1
    for (int ch = 0; ch < OZ_EPI_COLS; ch += 2) {
        int32_t v[OZ_MAX_DIGITS][2];
        oz_drain2(taddr + (uint32_t)ch, nd, v);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (ch + c >= ncol) continue;
            long long w[4];
            oz_groups(v, c, w);
            const int e = ei + ej[ch + c];
            const dd_t res = oz_sub(ct[(ch + c) * OZ_ROWS_A], ldexp((double)w[0], e - 40), ldexp((double)w[1], e - 72), ldexp((double)w[2], e - 104),
                                    ldexp((double)w[3], e - 136));
            __stcs(reinterpret_cast<double2 *>(cp + ldc * (long)(ch + c)), make_double2(res.hi, res.lo));
        }
    }
}

// Epilogue warps 1-16: warp w reads tensor-memory lanes 32 (w mod 4) .. +31
// (its rows of the tile) and columns 4 h .. 4 h + 3 of every diagonal,
// h = (w - 1) / 4, two columns at a time with all diagonals in one round
// trip, joins each entry's diagonals to four integers and subtracts them from
// C, whose tile lies in shared memory.
// FP64 and tensor instructions share a pipe of the SM: the FP64 part of a
// tile takes 1.5k cycles without MMAs, 2.9k beside them.  So the digits meet
// in the integer units (35 FP64 instructions an entry remain of 53), and an
// accumulator buffer goes back only after the tile's FP64 part, not when it
// is drained: the MMAs of the tile after next then run while the warps wait,
// drain and join the next tile (n = 9920, 14 digits: 451 us against 494).
// NDC: the digit count when known at compile time, else 0.
template <int NDC>
__device__ void oz_epilogue(const OzArgs &a, OzShared &S, const uint8_t *smC, int I, int J, int ntile) {
    volatile int *abort_flag = &S.abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = warp & 3, h = (warp - 1) >> 2;
    const int row = 32 * q + lane;
    const uint32_t lane_base = S.tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(OZ_EPI_COLS * h);
    const double2 *ct0 = reinterpret_cast<const double2 *>(smC) + (OZ_EPI_COLS * h) * OZ_ROWS_A + row;
    const int nd = NDC > 0 ? NDC : a.nd; // diagonals 2 .. B+1
    // the warp goes on together (the tensor-memory loads are warp-collective)
    auto wait_warp = [&](uint64_t *bar, uint32_t parity, int code) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        return oz_wait_lane0(bar, parity, abort_flag, a.err, code, a.wait_ns);
    };
    int st = 0; // done[] stage and parity of tile n
    uint32_t ph = 0;
    // scale exponents of tile n's row (padded rows hold 0) and columns
    int ei = 0;
    int4 ej = make_int4(0, 0, 0, 0);
    auto load_exps = [&]() {
        ei = a.exps[I * OZ_ROWS_A + row];
        ej = *reinterpret_cast<const int4 *>(a.exps + J * OZ_COLS_B + OZ_EPI_COLS * h);
    };
    load_exps();
    for (int n = 0; n < ntile; ++n) {
        const int i = I * OZ_ROWS_A + row;
        const int jb = J * OZ_COLS_B + OZ_EPI_COLS * h;
        const int b = n & 1, cs = n % OZ_C_STAGES;
        dd_t *cp = a.C + i + a.ldc * (long)jb;
        // entries of the lower triangle of C: columns jb .. jb + ncol - 1
        const int ncol = (i < a.n && i >= a.skip) ? max(0, min(OZ_EPI_COLS, min(a.n, i + 1) - jb)) : 0;
        const int e[4] = {ei + ej.x, ei + ej.y, ei + ej.z, ei + ej.w};
        const int eic = ei, *ejc = a.exps + jb;
        // every scale well inside the exponent range
        const bool mid = min(min(e[0], e[1]), min(e[2], e[3])) >= -900 && max(max(e[0], e[1]), max(e[2], e[3])) <= 1000;
        oz_tile_next(a.nJ, I, J);
        if (n + 1 < ntile) load_exps();
        if (!wait_warp(&S.cfull[cs], (uint32_t)((n / OZ_C_STAGES) & 1), 8)) break;
        const double2 *ct = ct0 + cs * (OZ_C_BYTES / 16);
        const uint32_t tb = lane_base + (uint32_t)(b * OZ_ACC_COLS);
        if (__all_sync(0xffffffffu, mid)) {
            double2 cv[OZ_EPI_COLS];
#pragma unroll
            for (int c = 0; c < OZ_EPI_COLS; ++c) cv[c] = c < ncol ? ct[c * OZ_ROWS_A] : make_double2(0.0, 0.0);
            if (!wait_warp(&S.done[st], ph, 6)) break;
            tc_fence_after();
            long long w[OZ_EPI_COLS][4];
#pragma unroll
            for (int ch = 0; ch < OZ_EPI_COLS; ch += 2) {
                int32_t v[OZ_MAX_DIGITS][2];
                oz_drain2(tb + (uint32_t)ch, nd, v);
#pragma unroll
                for (int c = 0; c < 2; ++c) oz_groups(v, c, w[ch + c]);
            }
#pragma unroll
            for (int c = 0; c < OZ_EPI_COLS; ++c) {
                const int k = 0x43380000 + (e[c] - 40) * 0x100000;
                const dd_t res = oz_sub(cv[c], oz_scaled(w[c][0], k), oz_scaled(w[c][1], k - 32 * 0x100000), oz_scaled(w[c][2], k - 64 * 0x100000),
                                        oz_scaled(w[c][3], k - 96 * 0x100000));
                if (c < ncol) __stcs(reinterpret_cast<double2 *>(cp + a.ldc * (long)c), make_double2(res.hi, res.lo));
            }
        } else {
            if (!wait_warp(&S.done[st], ph, 6)) break;
            tc_fence_after();
            oz_tile_far(tb, nd, ct, cp, a.ldc, ncol, eic, ejc);
        }
        // the buffer goes back only now: see above
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&S.tempty[b]);
            mbar_arrive(&S.cempty[cs]);
        }
        if (++st == OZ_STAGES) {
            st = 0;
            ph ^= 1u;
        }
    }
}

__global__ void __maxnreg__(OZ_MAX_REGS) ozaki_syrk_kernel(OzArgs a) {
    extern __shared__ uint8_t oz_raw[];
    __shared__ OzShared S;
    uint8_t *smA = reinterpret_cast<uint8_t *>(((uintptr_t)oz_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *smB = smA + (size_t)OZ_MAX_DIGITS * OZ_A_BYTES;
    uint8_t *smC = smB + (size_t)OZ_STAGES * OZ_TILE_B;
    const int tid = threadIdx.x, warp = tid >> 5;
    const long t_begin = a.tiles * blockIdx.x / gridDim.x, t_end = a.tiles * (blockIdx.x + 1) / gridDim.x;
    if (t_begin >= t_end) return;
    if (tid == 0) {
        S.abort_flag = *(volatile int *)a.err != 0;
        mbar_init(&S.barA, 1);
        mbar_init(&S.fin, 1);
        for (int st = 0; st < OZ_STAGES; ++st) {
            mbar_init(&S.barB[st], 1);
            mbar_init(&S.done[st], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&S.tempty[b], OZ_EPI_WARPS);
        }
        for (int st = 0; st < OZ_C_STAGES; ++st) {
            mbar_init(&S.cfull[st], 1);
            mbar_init(&S.cempty[st], OZ_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (S.abort_flag) return;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    int I, J;
    oz_tile_at(t_begin, a.nI, a.nJ, I, J);
    const int ntile = (int)(t_end - t_begin);
    if (warp == 0) {
        if ((tid & 31) == 0) oz_mma(a, S, smA, smB, I, J, ntile);
        __syncwarp();
    } else if (warp == OZ_AB_WARP) {
        oz_load_ab(a, S, smA, smB, I, J, ntile);
    } else if (warp == OZ_C_WARP) {
        oz_load_c(a, S, smC, I, J, ntile);
    } else {
        if (a.nd == OZ_MAX_DIGITS)
            oz_epilogue<OZ_MAX_DIGITS>(a, S, smC, I, J, ntile);
        else
            oz_epilogue<0>(a, S, smC, I, J, ntile);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(512) : "memory");
    }
}

// |x| 2^(120-e) truncated to an integer, with x's sign, for |x| 2^-e < 1/2:
// the significand of x (53 bits) shifted.  A value that is not finite gives 0.
__device__ __forceinline__ __int128 oz_fixed(double x, int e) {
    const long long bits = __double_as_longlong(x);
    const int ex = (int)((bits >> 52) & 0x7ff);
    if (ex == 0x7ff) return 0;
    const unsigned long long m = (unsigned long long)(bits & 0xfffffffffffffll) | (ex ? 1ull << 52 : 0ull);
    const int q = max(ex, 1) - 1075 + 120 - e;
    unsigned __int128 u = 0;
    if (q >= 0) u = (unsigned __int128)m << min(q, 127);
    else if (q > -64) u = m >> -q;
    return bits < 0 ? -(__int128)u : (__int128)u;
}

// Byte k of four words, for k = 0..3: a 4 x 4 byte transpose.
__device__ __forceinline__ void oz_transpose4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t *o) {
    const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
    o[0] = __byte_perm(ab0, cd0, 0x5410);
    o[1] = __byte_perm(ab0, cd0, 0x7632);
    o[2] = __byte_perm(ab1, cd1, 0x5410);
    o[3] = __byte_perm(ab1, cd1, 0x7632);
}

// Digits of 32 rows per CTA; warp c takes K bytes 16c..16c+15.  An entry is
// a 120-bit fixed-point integer U = P(r,k) 2^(120-e); with 128 added to the
// bytes of digits 1 .. nd and to the next lower one, if there is one (the rounding
// of the last digit), the bytes are the digits plus 128.
// A digit after the other peeled in dd arithmetic (10 FP64 operations each)
// and written in two layouts took 14.6 us at n = 5003; this takes 6.8.
__global__ void __launch_bounds__(128) ozaki_split_kernel(const dd_t *P, long ldp, int n, int k, int nd, int8_t *digits, int *exps) {
    __shared__ double rmax[4][32];
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    const int r = blockIdx.x * 32 + lane;
    dd_t x[16];
    double m = 0.0;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int kk = 16 * c + q;
        x[q] = (r < n && kk < k) ? ld_dd(P + r + ldp * (long)kk) : dd_zero();
        m = fmax(m, fabs(x[q].hi));
    }
    rmax[c][lane] = m;
    __syncthreads();
    m = fmax(fmax(rmax[0][lane], rmax[1][lane]), fmax(rmax[2][lane], rmax[3][lane]));
    int e = 0;
    if (m > 0.0) {
        int E;
        const double f = frexp(m, &E); // m = f 2^E, 1/2 <= f < 1
        e = E + (f > 0.996 ? 2 : 1);   // |P| 2^-e <= 0.498
    }
    if (c == 0) exps[r] = e;
    // byte p (0 .. 14) holds digit 15 - p: bytes 14 .. 15 - nd and one below
    unsigned __int128 bias = 0;
    for (int p = 14; p >= max(0, 14 - nd); --p) bias |= (unsigned __int128)0x80u << (8 * p);
    uint32_t w[4][16]; // w[j][q]: word j of value q, its bytes the digits plus 128
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const unsigned __int128 u = (unsigned __int128)(oz_fixed(x[q].hi, e) + oz_fixed(x[q].lo, e)) + bias;
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j][q] = (uint32_t)(u >> (32 * j)) ^ 0x80808080u;
    }
    const int within = ((r >> 3) & 1) * 512 + c * 128 + (r & 7) * 16; // offset inside a 16-row block of one digit
    int8_t *dst = digits + (long)(r >> 4) * nd * 1024 + within;
#pragma unroll
    for (int j = 3; j >= 0; --j) {
        uint32_t o[4][4]; // o[g][b]: byte b of the word of values 4g .. 4g+3
#pragma unroll
        for (int g = 0; g < 4; ++g) oz_transpose4(w[j][4 * g], w[j][4 * g + 1], w[j][4 * g + 2], w[j][4 * g + 3], o[g]);
#pragma unroll
        for (int b = 3; b >= 0; --b) {
            const int s = 15 - (4 * j + b); // digit
            if (s >= 1 && s <= nd) *reinterpret_cast<uint4 *>(dst + (long)(s - 1) * 1024) = make_uint4(o[0][b], o[1][b], o[2][b], o[3][b]);
        }
    }
}

} // namespace

void ozaki_syrk_sub_lower(cudaStream_t st, const dd_t *P, long ldp, int n, int k, dd_t *C, long ldc, OzakiWork &w, int skip, int reserve_sms) {
    if (n <= 0 || k <= 0) return;
    if (k > OZ_K) throw Error(ERR_ARG, "ozaki: panel wider than 64 columns");
    if (w.slices_used < 8 || w.slices_used > OZ_MAX_SLICES) throw Error(ERR_ARG, "ozaki: slice count must be 8..16");
    const int rows = (int)(ceil_div(n, OZ_ROWS_A) * OZ_ROWS_A);
    if (rows > w.row_cap || !w.digits || !w.exps || !w.err) throw Error(ERR_ARG, "ozaki: workspace smaller than the panel");
    const int nd = ozaki_digits(w.slices_used);
    ozaki_split_kernel<<<rows / 32, 128, 0, st>>>(P, ldp, n, k, nd, w.digits, w.exps);
    CK_LAUNCH();
    OzArgs a;
    a.digits = w.digits;
    a.exps = w.exps;
    a.C = C;
    a.ldc = ldc;
    a.n = n;
    a.nd = nd;
    a.nI = rows / OZ_ROWS_A;
    a.nJ = (int)ceil_div(n, OZ_COLS_B);
    a.skip = skip;
    a.err = w.err;
    a.wait_ns = w.wait_ns;
    long tiles = 0;
    for (int I = 0; I < a.nI; ++I) tiles += std::min((long)(OZ_ROWS_A / OZ_COLS_B) * (I + 1), (long)a.nJ);
    a.tiles = tiles;
    static thread_local int sms[64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int &sm = sms[dev & 63];
    if (sm == 0) {
        CK(cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev));
        CK(cudaFuncSetAttribute(ozaki_syrk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM));
    }
    const int grid = (int)std::min<long>(std::max(1, sm - reserve_sms), tiles);
    ozaki_syrk_kernel<<<grid, OZ_THREADS, OZ_SMEM, st>>>(a);
    CK_LAUNCH();
}

void ozaki_check(cudaStream_t st, const OzakiWork &w) {
    if (!w.err) return;
    int err = 0;
    int *h = w.h_err ? w.h_err : &err;
    CK(cudaMemcpyAsync(h, w.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (w.wait_ev) {
        CK(cudaEventRecord(w.wait_ev, st));
        CK(cudaEventSynchronize(w.wait_ev));
    } else {
        CK(cudaStreamSynchronize(st));
    }
    err = *h;
    if (err != 0) {
        // clear the error word, so that the next launch starts afresh
        CK(cudaMemsetAsync(w.err, 0, sizeof(int), st));
        CK(cudaStreamSynchronize(st));
        throw Error(ERR_CUDA, "ozaki: a tensor-core split update gave up waiting (code " + std::to_string(err) + ")");
    }
}

} // namespace sddd
