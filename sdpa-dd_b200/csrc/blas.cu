// Dense dd linear algebra on the FP64 pipe of sm_100a.
//
// Every kernel here reproduces the per-entry operation order of the
// MPLAPACK routine it replaces, so that with the same inputs it returns the
// reference's dd results bit for bit:
//   gemm       Rgemm_{NN,TN,NT}_omp  (mplapack/Rgemm_*_omp.cpp): each C(i,j)
//              is a sequential sum over k of "c += a*b" steps
//   potrf      Rpotrf("Lower") (mplapack/Rpotrf.cpp:124-142 with Rsyrk,
//              Rgemm, Rtrsm, Rpotrf2): entry (i,j) receives the products
//              L(j,k)L(i,k) for k ascending as "x = x - p" steps, the diagonal
//              takes sqrt and the column below is scaled by 1/L(j,j)
//   trsv       Rtrsv("Lower", "N"/"T", "NonUnit") (mplapack/Rtrsv.cpp)
//   inv_lower  Rtrsm("Left","Lower","N","N") on the identity
//              (Lal::getInvLowTriangularMatrix, sdpa_linear.cpp:397-412)
//   trmm_lt    Rtrmm("Left","Lower","Transpose","NonUnit")
//              (Jal::getInvCholAndInv, sdpa_jordan.cpp:154-170)
//   symmetrize Lal::getSymmetrize (sdpa_linear.cpp:414-438)
// The blocking below (tiles, panels) is the B200 schedule; it never
// reorders the operations that land on one entry.
#include "blas.h"
#include "bulk.cuh"
#include "devops.cuh"
#include "fastdiv.cuh"
#include "ozaki.h"
#include "prof.h"
#include "tile16.cuh"

#include <algorithm>

namespace sddd {

// ===================================================================== GEMM
// Tile: BM x BN outputs per CTA, BK-deep k slices staged in shared memory,
// TM x TN outputs per thread.  Shared tiles are k-major and padded by one
// element so that transposed tile loads do not collide on banks.
// beta C(i,j) as Rgemm's first loop leaves it: zero for beta == 0, unchanged
// for beta == 1, else beta * C(i,j).
__device__ __forceinline__ dd_t beta_times(dd_t beta, const dd_t *cp) {
    if (dd_is_zero(beta)) return dd_zero();
    const dd_t c = ld_dd(cp);
    return beta.hi == 1.0 && beta.lo == 0.0 ? c : dd_mul(beta, c);
}
// MODE GEMM_AB_PRE (Rgemm_NN/NT_omp with alpha): each B value is multiplied
// by alpha as it is staged ("temp = alpha * B(l,j)"), then c += temp * a
// from the (beta-scaled) C; GEMM_AB_POST (Rgemm_TN/TT_omp): the products
// are summed from zero and C += alpha * sum.
// STACK: the rows of A and C are those of M / stack matrices of `stack` rows,
// one after the other, matrix r at A + r sA and C + r sC.
template <int BM, int BN, int BK, int TM, int TN, bool TA, bool TB, int MODE, bool STACK = false>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    gemm_kernel(int M, int N, int K, const dd_t *__restrict__ A, long lda, long sA, const dd_t *__restrict__ B, long ldb, long sB, dd_t *C,
                long ldc, long sC, int lower, dd_t alpha, dd_t beta, int stack) {
    static_assert(!STACK || (!TA && MODE == GEMM_STORE), "the stacked form is A_r B");
    constexpr int TX = BN / TN, TY = BM / TM, NT = TX * TY;
    __shared__ double2 As[BK][BM + 1];
    __shared__ double2 Bs[BK][BN + 1];
    __shared__ long arow[STACK ? BM : 1]; // a row's offset in A
    const long bz = blockIdx.z;
    if (!STACK) {
        A += bz * sA;
        C += bz * sC;
    }
    B += bz * sB;
    // (the long dimension of a stacked product is on grid.x)
    const int i0 = (STACK ? blockIdx.x : blockIdx.y) * BM, j0 = (STACK ? blockIdx.y : blockIdx.x) * BN;
    if (lower && i0 + BM <= j0) return; // tile entirely above the diagonal
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    if (STACK) {
        for (int e = tid; e < BM; e += NT) arow[e] = (i0 + e) / stack * sA + (i0 + e) % stack;
        __syncthreads();
    }
    dd_t acc[TM][TN];
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int c = 0; c < TN; ++c) {
            int gi = i0 + ty + TY * r, gj = j0 + tx + TX * c;
            if (MODE == GEMM_STORE || MODE == GEMM_AB_POST || gi >= M || gj >= N)
                acc[r][c] = dd_zero();
            else
                acc[r][c] = MODE == GEMM_AB_PRE ? beta_times(beta, C + gi + ldc * (long)gj) : ld_dd(C + gi + ldc * (long)gj);
        }
    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int e = tid; e < BM * BK; e += NT) {
            int ii, kk;
            if (!TA) {
                ii = e % BM;
                kk = e / BM;
            } else {
                kk = e % BK;
                ii = e / BK;
            }
            int gi = i0 + ii, gk = k0 + kk;
            double2 v = make_double2(0.0, 0.0);
            if (gi < M && gk < K) v = *reinterpret_cast<const double2 *>(TA ? A + gk + lda * (long)gi : A + (STACK ? arow[ii] : gi) + lda * (long)gk);
            As[kk][ii] = v;
        }
        for (int e = tid; e < BN * BK; e += NT) {
            int jj, kk;
            if (!TB) {
                kk = e % BK;
                jj = e / BK;
            } else {
                jj = e % BN;
                kk = e / BN;
            }
            int gj = j0 + jj, gk = k0 + kk;
            double2 v = make_double2(0.0, 0.0);
            if (gj < N && gk < K) v = *reinterpret_cast<const double2 *>(TB ? B + gj + ldb * (long)gk : B + gk + ldb * (long)gj);
            if (MODE == GEMM_AB_PRE) {
                const dd_t t = dd_mul(alpha, dd_make(v.x, v.y));
                v = make_double2(t.hi, t.lo);
            }
            Bs[kk][jj] = v;
        }
        __syncthreads();
        const int kmax = min(BK, K - k0);
        for (int kk = 0; kk < kmax; ++kk) {
            dd_t a[TM], b[TN];
#pragma unroll
            for (int r = 0; r < TM; ++r) {
                double2 v = As[kk][ty + TY * r];
                a[r] = dd_make(v.x, v.y);
            }
#pragma unroll
            for (int c = 0; c < TN; ++c) {
                double2 v = Bs[kk][tx + TX * c];
                b[c] = dd_make(v.x, v.y);
            }
#pragma unroll
            for (int r = 0; r < TM; ++r)
#pragma unroll
                for (int c = 0; c < TN; ++c) {
                    dd_t p = dd_mul(b[c], a[r]);
                    acc[r][c] = (MODE == GEMM_SUB) ? dd_sub(acc[r][c], p) : dd_acc(acc[r][c], p);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int c = 0; c < TN; ++c) {
            int gi = i0 + ty + TY * r, gj = j0 + tx + TX * c;
            if (gi < M && gj < N && (!lower || gi >= gj)) {
                dd_t *cp = C + (STACK ? gi / stack * sC + gi % stack : gi) + ldc * (long)gj;
                st_dd(cp, MODE == GEMM_AB_POST ? dd_acc(beta_times(beta, cp), dd_mul(alpha, acc[r][c])) : acc[r][c]);
            }
        }
}

// The same in 16 x 16 tiles (tile16.cuh).  Order 500: 183 us in isolation, the
// FP64 work alone 134; one entry a thread, 256 threads, took 204 (a call of that
// order, with its launch and wait, 224 and 228).
template <bool TA, bool TB, int MODE, bool PIPE>
__global__ void __launch_bounds__(T16_THREADS, T16_CTAS)
    gemm16_kernel(int M, int N, int K, const dd_t *__restrict__ A, long lda, long sA, const dd_t *__restrict__ B, long ldb, long sB, dd_t *C, long ldc,
                  long sC, int lower, dd_t alpha, dd_t beta) {
    __shared__ Tile16 S;
    const long bz = blockIdx.z;
    A += bz * sA;
    B += bz * sB;
    C += bz * sC;
    const int i0 = blockIdx.y * T16, j0 = blockIdx.x * T16;
    if (lower && i0 + T16 <= j0) return; // tile entirely above the diagonal
    const int gj = j0 + threadIdx.x % T16, gi = i0 + threadIdx.x / T16;
    dd_t acc[2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (MODE == GEMM_STORE || MODE == GEMM_AB_POST || gi + 8 * r >= M || gj >= N)
            acc[r] = dd_zero();
        else
            acc[r] = MODE == GEMM_AB_PRE ? beta_times(beta, C + gi + 8 * r + ldc * (long)gj) : ld_dd(C + gi + 8 * r + ldc * (long)gj);
    tile16_sum<TA, !TB, MODE == GEMM_SUB, PIPE>(
        S, K,
        [&](int i, long k) {
            return i0 + i < M ? *reinterpret_cast<const double2 *>(TA ? A + k + lda * (long)(i0 + i) : A + i0 + i + lda * k) : make_double2(0.0, 0.0);
        },
        [&](int j, long k) {
            if (j0 + j >= N) return make_double2(0.0, 0.0);
            const double2 v = *reinterpret_cast<const double2 *>(TB ? B + j0 + j + ldb * k : B + k + ldb * (long)(j0 + j));
            if (MODE != GEMM_AB_PRE) return v;
            const dd_t t = dd_mul(alpha, dd_make(v.x, v.y));
            return make_double2(t.hi, t.lo);
        },
        acc);
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (gi + 8 * r < M && gj < N && (!lower || gi + 8 * r >= gj)) {
            dd_t *cp = C + gi + 8 * r + ldc * (long)gj;
            st_dd(cp, MODE == GEMM_AB_POST ? dd_acc(beta_times(beta, cp), dd_mul(alpha, acc[r])) : acc[r]);
        }
}

// 64 x 64 tiles (4 x 4 entries a thread) when they fill the GPU; 16 x 16
// tiles for small products (fewer 64 x 64 tiles than half the SMs), so that
// the work spreads over more SMs, and where the larger tiles would be mostly
// padding (16 x 16 tiles run at about 0.7 of the FP64 rate, 64 x 64 at 0.9;
// 200 products of order 20: 33 us in 64 x 64 tiles,
// 9 in 16 x 16).  A launch has at most MAX_GRID_YZ tiles down, 1,048,560 rows of
// 16 x 16 tiles; taller products keep the 64 x 64 ones.  Each entry's k-order is
// the same either way.
constexpr long GEMM_SMALL_TILES = 74;
template <bool TA, bool TB, int MODE>
static void gemm_launch(cudaStream_t st, int M, int N, int K, const dd_t *A, long lda, long sA, const dd_t *B, long ldb, long sB, dd_t *C, long ldc,
                        long sC, int batch, bool lower, dd_t alpha = dd_t{1.0, 0.0}, dd_t beta = dd_t{1.0, 0.0}) {
    const long m16 = ceil_div(M, T16), n16 = ceil_div(N, T16), m64 = ceil_div(M, 64), n64 = ceil_div(N, 64);
    if (m16 <= MAX_GRID_YZ && (m64 * n64 * batch < GEMM_SMALL_TILES || 13 * m16 * n16 < 10 * 16 * m64 * n64)) {
        dim3 grid((unsigned)n16, (unsigned)m16, batch);
        if (m16 * n16 * batch <= T16_PIPE_TILES)
            gemm16_kernel<TA, TB, MODE, true><<<grid, T16_THREADS, 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, lower ? 1 : 0, alpha, beta);
        else
            gemm16_kernel<TA, TB, MODE, false><<<grid, T16_THREADS, 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, lower ? 1 : 0, alpha, beta);
        CK_LAUNCH();
        return;
    }
    constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
    dim3 grid((unsigned)n64, (unsigned)m64, batch);
    gemm_kernel<BM, BN, BK, TM, TN, TA, TB, MODE>
        <<<grid, (BM / TM) * (BN / TN), 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, lower ? 1 : 0, alpha, beta, 0);
    CK_LAUNCH();
}

// C_r = A_r B (rows) or C_r = A B_r of `count` matrices of order n that lie
// n^2 apart, as one product whose long dimension runs through the matrices,
// so that only the other one is padded; its tile is 4 TS wide, TS threads of
// four entries, TS as the order wants it.
template <int TS> static void stacked_launch(cudaStream_t st, bool rows, int n, int count, const dd_t *A, const dd_t *B, dd_t *C) {
    constexpr int BS = 4 * TS, BL = 64, BK = 16;
    const long nn = (long)n * n;
    const dd_t one = {1.0, 0.0};
    const unsigned tl = ceil_div((long)n * count, BL), ts = ceil_div(n, BS);
    if (rows)
        gemm_kernel<BL, BS, BK, 4, 4, false, false, GEMM_STORE, true>
            <<<dim3(tl, ts), 16 * TS, 0, st>>>(n * count, n, n, A, n, nn, B, n, 0, C, n, nn, 0, one, one, n);
    else
        gemm_kernel<BS, BL, BK, 4, 4, false, false, GEMM_STORE>
            <<<dim3(tl, ts), 16 * TS, 0, st>>>(n, n * count, n, A, n, 0, B, n, 0, C, n, 0, 0, one, one, 0);
    CK_LAUNCH();
}
void gemm_stacked(cudaStream_t st, bool rows, int n, int count, const dd_t *A, const dd_t *B, dd_t *C) {
    if (n <= 0 || count <= 0) return;
    // the fewest warps over the short dimension, then the fewest tiles (an odd
    // width has as many warps as the next even one)
    int ts = 8, best = 1 << 30;
    for (int t = 16; t >= 8; t -= 2) {
        const int tiles = (int)ceil_div(n, 4 * t), cost = tiles * (int)ceil_div(16 * t, 32);
        if (cost < best) best = cost, ts = t;
    }
    const long nn = (long)n * n;
    if ((long)n * count > (1L << 30) || (long)ceil_div((long)n * count, 64) * ceil_div(n, 4 * ts) < 2 * GEMM_SMALL_TILES) {
        gemm(st, 'N', 'N', GEMM_STORE, n, n, n, A, n, rows ? nn : 0, B, n, rows ? 0 : nn, C, n, nn, count, false);
        return;
    }
    switch (ts) {
    case 8: stacked_launch<8>(st, rows, n, count, A, B, C); break;
    case 10: stacked_launch<10>(st, rows, n, count, A, B, C); break;
    case 12: stacked_launch<12>(st, rows, n, count, A, B, C); break;
    case 14: stacked_launch<14>(st, rows, n, count, A, B, C); break;
    default: stacked_launch<16>(st, rows, n, count, A, B, C);
    }
}

// C = beta C alone (a product without terms).
__global__ void gemm_beta_kernel(dd_t *C, long ldc, int M, int N, dd_t beta) {
    const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)M * N) return;
    dd_t *cp = C + e % M + ldc * (e / M);
    st_dd(cp, beta_times(beta, cp));
}

void gemm_ab(cudaStream_t st, char ta, char tb, int M, int N, int K, dd_t alpha, const dd_t *A, long lda, const dd_t *B, long ldb, dd_t beta, dd_t *C,
             long ldc) {
    const bool one_beta = beta.hi == 1.0 && beta.lo == 0.0;
    const bool zero_alpha = alpha.hi == 0.0 && alpha.lo == 0.0;
    if (M <= 0 || N <= 0 || ((zero_alpha || K <= 0) && one_beta)) return; // Rgemm's quick return
    if (zero_alpha || K <= 0) {
        gemm_beta_kernel<<<ceil_div((long)M * N, 256), 256, 0, st>>>(C, ldc, M, N, beta);
        CK_LAUNCH();
        return;
    }
    const bool a = ta == 'T', b = tb == 'T';
    if (!a && !b) gemm_launch<false, false, GEMM_AB_PRE>(st, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, false, alpha, beta);
    else if (!a && b) gemm_launch<false, true, GEMM_AB_PRE>(st, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, false, alpha, beta);
    else if (a && !b) gemm_launch<true, false, GEMM_AB_POST>(st, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, false, alpha, beta);
    else gemm_launch<true, true, GEMM_AB_POST>(st, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, false, alpha, beta);
}

void gemm(cudaStream_t st, char ta, char tb, int mode, int M, int N, int K, const dd_t *A, long lda, long sA, const dd_t *B, long ldb, long sB,
          dd_t *C, long ldc, long sC, int batch, bool lower) {
    if (M <= 0 || N <= 0 || batch <= 0) return;
    if (K <= 0 && mode == GEMM_SUB) return;
    if (batch > MAX_GRID_YZ) {
        // grid.z holds at most 65535 matrices per launch
        for (int b0 = 0; b0 < batch; b0 += MAX_GRID_YZ)
            gemm(st, ta, tb, mode, M, N, K, A + b0 * sA, lda, sA, B + b0 * sB, ldb, sB, C + b0 * sC, ldc, sC, std::min(MAX_GRID_YZ, batch - b0), lower);
        return;
    }
#define GL(TA_, TB_, MD_) gemm_launch<TA_, TB_, MD_>(st, M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, lower)
    bool a = ta == 'T', b = tb == 'T';
    if (mode == GEMM_STORE) {
        if (!a && !b) GL(false, false, GEMM_STORE);
        else if (a && !b) GL(true, false, GEMM_STORE);
        else if (!a && b) GL(false, true, GEMM_STORE);
        else GL(true, true, GEMM_STORE);
    } else if (mode == GEMM_SUB) {
        if (!a && b) GL(false, true, GEMM_SUB);
        else if (!a && !b) GL(false, false, GEMM_SUB);
        else throw Error(ERR_ARG, "gemm: unsupported SUB variant");
    } else {
        if (!a && !b) GL(false, false, GEMM_ACC);
        else if (a && !b) GL(true, false, GEMM_ACC);
        else throw Error(ERR_ARG, "gemm: unsupported ACC variant");
    }
#undef GL
}

// ==================================================================== POTRF
// Diagonal block: right-looking dd Cholesky of an nb x nb block, nb <= 64.
// On a non-positive or NaN pivot the 1-based global column goes to *info
// and the block is left as it was (Rpotrf2's n = 1 test,
// mplapack/Rpotrf2.cpp).  1/L(j,j) for the panel goes to rdiag.
//
// The block's time is its chain of pivots (a dd square root and reciprocal, a
// product and a subtraction a column), so warp 0 carries that chain, alone on
// its SM sub-partition (warps 4, 8, .. have no work): with column k in
// registers (lane i holds rows i and i + 32), its last term still to come, it
// forms L(k,k) and 1/L(k,k) in all lanes and that term beside them, takes
// column k + 1, forms the next pivot from L(k+1,k) = x(k+1,k) / L(k,k) in
// every lane, and scales and publishes column k beside that.  The warps of the
// other sub-partitions hold columns 2 .. nb-1 in registers, in pairs j + j' =
// nb + 2 whose nb - 2 entries fill two slots a lane, subtract the published
// columns' terms, and hand column j over once column j - 2's term is in.
// Hand-overs are named barriers, which have no time limit: a warp that waits at
// one is freed only by the other warps' arrivals, so no warp may leave by
// itself.  The whole CTA decides on one read of *info whether it runs (other
// CTAs of a batch write that word at any time); on a bad pivot k warp 0 still
// publishes column k, so the helpers, which wait for published columns only, see
// the stop there and end too (the hand-over of column k + 1, which its helper may
// have signalled, is then waited for by nobody; an arrival does not wait).
// Every entry sees x(i,j) -= L(j,k) L(i,k) for k ascending, then the sqrt or the
// scaling.
// Measured for nb = 64: 46 us; with warps that took turns at the pivot, on
// lane 0 and with the plain divisions, behind an mbarrier a column, 70 us.
// The same behind mbarriers 57 us (a wake-up costs several hundred cycles),
// behind polled flags 53 us (the polls take the issue slots of the warps at
// work); a second warp for the columns 52 us (their hand-over waits for the
// helpers' FP64 work either way); sub-blocks of 16 columns in warp 0's
// registers 95 us.
constexpr int DIAG_THREADS = 1024;
constexpr int DIAG_HELPERS = 24;
constexpr int DIAG_PAIRS = 2;   // pairs a helper holds at most
constexpr unsigned long long POTRF_WAIT_NS = 2000000000ull; // one wait, at most
static_assert(POTRF_NB <= 64 && DIAG_THREADS == 1024 && DIAG_HELPERS * DIAG_PAIRS >= POTRF_NB / 2, "two rows a lane; warps 1-3, 5-7, .. help");
__device__ __forceinline__ dd_t shfl_dd(dd_t v, int src) {
    return dd_make(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
// Bounded wait for phase 0 of an mbarrier.
__device__ __forceinline__ bool bar_wait0(uint64_t *b) {
    if (mbar_try_wait(b, 0)) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (!mbar_try_wait(b, 0))
        if (globaltimer_ns() - t0 > POTRF_WAIT_NS) return false;
    return true;
}
template <int NB>
__device__ __forceinline__ void potrf_diag_body(dd_t *A, long lda, int nb_, int c0, int *info, dd_t *rdiag) {
    const int nb = NB > 0 ? NB : nb_;
    extern __shared__ double2 sm[];
    double2 *S = sm; // nb x nb, column-major: columns on their way, then final
    __shared__ int skip, stop; // skip: a block before failed; stop: k + 1 for a bad pivot k
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        skip = *reinterpret_cast<volatile int *>(info);
        stop = 0;
    }
    for (int e = tid; e < nb * nb; e += DIAG_THREADS) {
        const int i = e % nb, j = e / nb;
        if (i >= j) {
            const dd_t v = ld_dd(A + (c0 + i) + lda * (long)(c0 + j));
            S[e] = make_double2(v.hi, v.lo);
        }
    }
    __syncthreads();
    if (skip != 0) return; // (written once: the same in every thread)
    volatile int *vstop = &stop;
    auto at = [&](int i, int j) {
        const double2 v = S[i + nb * j];
        return dd_make(v.x, v.y);
    };
    auto put = [&](int i, int j, dd_t v) { S[i + nb * j] = make_double2(v.hi, v.lo); };
    // Named barriers, four of a kind in turn (by k).  Column k published (k <
    // nb - 2): warp 0 arrives, the helpers wait, so none is a whole turn
    // behind.  Column k handed over (k >= 2): its helper arrives, warp 0 waits.
    auto bar_arrive = [](int id, int warps) {
        __syncwarp();
        asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(32 * warps) : "memory");
    };
    auto bar_wait = [](int id, int warps) {
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(32 * warps) : "memory");
    };
    auto column_id = [](int k) { return 1 + (k & 3); };
    auto handed_id = [](int k) { return 5 + (k & 3); };
    const int columns = nb - 2;
    if (warp == 0) {
        const int i0 = min(lane, nb - 1), i1 = min(lane + 32, nb - 1); // (a repeated last row is not stored)
        // column k is c - ln L(:, k - 1)
        dd_t ca = at(i0, 0), cb = at(i1, 0), ln = dd_zero(), la = ln, lb = ln, d = at(0, 0);
        for (int k = 0; k < nb; ++k) {
            if (dd_le_d(d, 0.0) || dd_isnan(d)) {
                if (lane == 0) {
                    *info = c0 + k + 1;
                    *vstop = k + 1; // the helpers stop at column k
                }
                if (k < columns) bar_arrive(column_id(k), 1 + DIAG_HELPERS);
                break;
            }
            const int kn = min(k + 1, nb - 1);
            dd_t l, r;
            const bool fast = sqrt_rcp_fast(d, l, r);
            // the column's last term, and its entry of the next row in every
            // lane, beside the pivot's chain
            const dd_t ua = dd_sub(ca, dd_mul(ln, la)), ub = dd_sub(cb, dd_mul(ln, lb));
            const dd_t xa = k > 0 ? ua : ca, xb = k > 0 ? ub : cb;
            const dd_t xn = shfl_dd(kn < 32 ? xa : xb, kn & 31);
            if (!fast) sqrt_rcp_plain(d, l, r);
            if (kn >= 2 && kn > k) bar_wait(handed_id(kn), 2);
            const dd_t dn = at(kn, kn);
            ca = at(i0, kn);
            cb = at(i1, kn);
            ln = dd_mul(r, xn);
            d = dd_sub(dn, dd_mul(ln, ln));
            la = lane == k ? l : dd_mul(r, xa);
            lb = lane + 32 == k ? l : dd_mul(r, xb);
            if (lane >= k && lane < nb) put(i0, k, la);
            if (lane + 32 >= k && lane + 32 < nb) put(i1, k, lb);
            if (lane == 0 && rdiag) st_dd(rdiag + k, r);
            if (k < columns) bar_arrive(column_id(k), 1 + DIAG_HELPERS);
        }
    } else if ((warp & 3) != 0) {
        const int h = (warp >> 2) * 3 + (warp & 3) - 1;
        // pair p: columns ja = 2 + p and jb = nb - p (none: -1); slot q of the
        // lane: entry q 32 + lane of the rows ja .. nb-1 of ja, then jb .. nb-1
        // of jb
        dd_t x[DIAG_PAIRS][2];
        int col[DIAG_PAIRS][2], row[DIAG_PAIRS][2], ja[DIAG_PAIRS], jb[DIAG_PAIRS];
#pragma unroll
        for (int c = 0; c < DIAG_PAIRS; ++c) {
            const int p = h + DIAG_HELPERS * c;
            ja[c] = 2 + p;
            jb[c] = nb - p;
            if (ja[c] > jb[c] || ja[c] >= nb) ja[c] = jb[c] = -1;
            if (jb[c] == ja[c] || jb[c] >= nb) jb[c] = -1;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = q * 32 + lane, na = ja[c] < 0 ? 0 : nb - ja[c];
                col[c][q] = e < na ? ja[c] : jb[c];
                row[c][q] = e < na ? ja[c] + e : jb[c] + e - na;
                if (col[c][q] < 0 || row[c][q] >= nb) col[c][q] = -1, row[c][q] = 0;
                x[c][q] = col[c][q] >= 0 ? at(row[c][q], col[c][q]) : dd_zero();
            }
        }
        for (int k = 0; k < columns; ++k) {
            bar_wait(column_id(k), 1 + DIAG_HELPERS);
            if (*vstop == k + 1) break;
            auto update = [&](const int c) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int j = col[c][q];
                    if (!__any_sync(0xffffffffu, j >= k + 2)) continue;
                    x[c][q] = dd_sub(x[c][q], dd_mul(at(max(j, k), k), at(max(row[c][q], k), k)));
                    if (j == k + 2) put(row[c][q], j, x[c][q]);
                }
                if (ja[c] == k + 2 || jb[c] == k + 2) bar_arrive(handed_id(k + 2), 2);
            };
            static_assert(DIAG_PAIRS == 2, "the urgent pair first");
            if (ja[1] == k + 2 || jb[1] == k + 2) {
                update(1);
                update(0);
            } else {
                update(0);
                update(1);
            }
        }
    }
    __syncthreads();
    if (stop != 0) return;
    for (int e = tid; e < nb * nb; e += DIAG_THREADS) {
        const int i = e % nb, j = e / nb;
        if (i >= j) st_dd(A + (c0 + i) + lda * (long)(c0 + j), at(i, j));
    }
}

// CTA b: matrix b of a batch of equal blocks (rdiag null then).
__global__ void __launch_bounds__(DIAG_THREADS) potrf_diag_kernel(dd_t *A, long lda, int nb, int c0, int *info, dd_t *rdiag, long sA) {
    if (nb == POTRF_NB) potrf_diag_body<POTRF_NB>(A + blockIdx.x * sA, lda, nb, c0, info, rdiag);
    else potrf_diag_body<0>(A + blockIdx.x * sA, lda, nb, c0, info, rdiag);
}
// CTA b: the block at column c0 of matrix b of a list (a kernel of its own:
// with the block's order and pointers in registers it takes 66 us, not 46).
__global__ void __launch_bounds__(DIAG_THREADS) potrf_diag_list_kernel(const PotrfItem *list, int c0) {
    const PotrfItem &it = list[blockIdx.x];
    if (c0 < it.n) potrf_diag_body<0>(it.A, it.n, min(POTRF_NB, it.n - c0), c0, it.info, it.rdiag);
}

// Panel rows below the diagonal block (Rtrsm "Right", "Lower", "Transpose":
// x(i,j) -= L(j,k) x(i,k) for k < j ascending, then x(i,j) *= 1/L(j,j)).
// Rows are independent, so a warp solves W = 32 / C rows by itself, with no
// barrier: lane = (column class c, row r), c = lane / W, and the lane holds the
// row's columns c, c + C, ... in registers.  At step k the holder of x(r,k)
// passes it to the row's other lanes by shuffle; every lane scales it (the
// entry is final; no branch for its holder) and subtracts the step's term from
// its columns right of k.
// Rounds of C steps: in round q, slot s holds column c + C (q + s) (the slots
// rotate by one between rounds, and the column leaving slot 0 is final and goes
// back to memory); the rounds are unrolled so that each one updates exactly its
// live slots, without branches between the slots' independent chains.  L11
// (lower triangle, packed by columns, one bulk copy per column) and the
// reciprocals are shared by the CTA's warps.  The panel is POTRF_NB columns
// wide.
// A step is a shuffle, a product, and a product and a subtraction (190
// cycles), or the FP64 issue of the live slots where there are rows enough.
// Measured (C = 16 / 8): 500 rows 14.0 / 15.4 us, 1500 16.9 / 15.8, 5000 35 /
// 31, 10000 58 / 48.6; with the holder scaling its entry under a branch and C =
// 16 18.5, 20.8, 37.5 and 60.
constexpr int PANEL_THREADS = 128;
// lanes a row -> rows a CTA
__host__ __device__ constexpr int panel_rows(int classes) { return 32 / classes * (PANEL_THREADS / 32); }
constexpr size_t PANEL_SMEM = sizeof(double2) * (POTRF_NB * (POTRF_NB + 1) / 2 + POTRF_NB);
// first entry of column k (rows k .. POTRF_NB-1) of a lower triangle packed
// by columns
__device__ __forceinline__ int col_off(int k) { return k * POTRF_NB - k * (k - 1) / 2; }
template <int PANEL_CLASSES>
__global__ void __launch_bounds__(PANEL_THREADS) potrf_panel_kernel(dd_t *A, long lda, int n, int c0, int *info, const dd_t *rdiag,
                                                                    const PotrfItem *list) {
    // lanes and columns a lane a row, rows a warp and a CTA
    constexpr int NB = POTRF_NB, C = PANEL_CLASSES, W = 32 / C, NS = NB / C, PANEL_ROWS = panel_rows(C);
    static_assert(NB % C == 0 && 32 % C == 0, "panel lane map");
    extern __shared__ __align__(16) double2 sm[];
    double2 *L11 = sm;                   // lower triangle of NB x NB, packed by columns
    double2 *R = sm + NB * (NB + 1) / 2; // NB reciprocals
    __shared__ uint64_t lbar;
    __shared__ int lfail;
    if (list) { // grid row y: matrix y of a list
        const PotrfItem &it = list[blockIdx.y];
        A = it.A;
        lda = n = it.n;
        info = it.info;
        rdiag = it.rdiag;
        if ((long)c0 + NB + (long)blockIdx.x * PANEL_ROWS >= n) return;
    }
    if (*info != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&lbar, 1);
        mbar_init_fence();
        lfail = 0;
    }
    __syncthreads();
    if (warp == 0) {
        // column k of L11 (rows k .. NB-1) is contiguous in A: one bulk copy
        if (lane == 0) mbar_expect_tx(&lbar, (uint32_t)(sizeof(double2) * NB * (NB + 1) / 2));
        __syncwarp();
        for (int k = lane; k < NB; k += 32)
            bulk_g2s(L11 + col_off(k), A + (c0 + k) + lda * (long)(c0 + k), (uint32_t)(sizeof(double2) * (NB - k)), &lbar);
    }
    for (int e = tid; e < NB; e += PANEL_THREADS) R[e] = make_double2(rdiag[e].hi, rdiag[e].lo);
    const int cls = lane / W, row = lane % W;
    const long gi = (long)c0 + NB + (long)blockIdx.x * PANEL_ROWS + warp * W + row;
    const bool live = gi < n;
    dd_t *arow = A + gi + lda * (long)c0; // the row's panel entries, stride lda
    dd_t x[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) x[s] = live ? ld_dd(arow + lda * (long)(cls + C * s)) : dd_from(0.0);
    if (tid == 0 && !bar_wait0(&lbar)) {
        // the copies did not land in time: report, let them land (bounded)
        lfail = 1;
        atomicCAS(info, 0, -1);
        bar_wait0(&lbar);
    }
    __syncthreads();
    if (lfail) return;
    auto rk = [&](int k) { return dd_make(R[k].x, R[k].y); };
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        // step k = C q + t; slot s holds column cls + C (q + s), s < NS - q
#pragma unroll 1
        for (int t = 0; t < C; ++t) {
            const int k = C * q + t;
            const double2 *lk = L11 + col_off(k) - k; // L(j, k) at lk[j]
            // x(r,k), final after its scaling, in all the row's lanes
            const dd_t xk = dd_mul(rk(k), dd_make(__shfl_sync(0xffffffffu, x[0].hi, t * W + row), __shfl_sync(0xffffffffu, x[0].lo, t * W + row)));
            dd_t y[NS];
#pragma unroll
            for (int s = 0; s < NS - q; ++s) {
                // (slot 0's columns left of k read some entry of L11, unused)
                const double2 l = lk[s == 0 ? max(cls + C * q, k) : cls + C * (q + s)];
                y[s] = dd_sub(x[s], dd_mul(dd_make(l.x, l.y), xk));
            }
            x[0] = cls > t ? y[0] : cls == t ? xk : x[0];
#pragma unroll
            for (int s = 1; s < NS - q; ++s) x[s] = y[s];
        }
        // column cls + C q is final
        if (live) st_dd(arow + lda * (long)(cls + C * q), x[0]);
#pragma unroll
        for (int s = 0; s + 1 < NS - q; ++s) x[s] = x[s + 1];
    }
}

// The next diagonal block's update by the panel just solved, ahead of the
// trailing update (the split form's lookahead): D(i, j) -= P(j, k) P(i, k)
// for k ascending, i >= j; CTA j takes column j, thread i row i.  D is the
// nb x nb block at c0, P its rows of the nbp panel columns before c0,
// staged in shared memory first (one bulk copy per panel column: its nb
// rows are contiguous) so that the chain of each entry reads no global
// memory.
__global__ void potrf_diag_pre_kernel(dd_t *A, long lda, int c0, int nb, int nbp, int *info) {
    extern __shared__ __align__(16) double2 pre_sp[]; // pre_sp[k * blockDim.x + r] = P(r, k)
    __shared__ uint64_t pbar;
    __shared__ int pfail;
    if (*info != 0) return;
    const int j = blockIdx.x, i = threadIdx.x, w = blockDim.x;
    const dd_t *P = A + c0 + lda * (long)(c0 - nbp);
    if (i == 0) {
        mbar_init(&pbar, 1);
        mbar_init_fence();
        pfail = 0;
    }
    __syncthreads();
    if (i < 32) {
        if (i == 0) mbar_expect_tx(&pbar, (uint32_t)(sizeof(double2) * nb * nbp));
        __syncwarp();
        for (int k = i; k < nbp; k += 32) bulk_g2s(pre_sp + k * w, P + lda * (long)k, (uint32_t)(sizeof(double2) * nb), &pbar);
    }
    if (i == 0 && !bar_wait0(&pbar)) {
        // the copies did not land in time: report, let them land (bounded)
        pfail = 1;
        atomicCAS(info, 0, -1);
        bar_wait0(&pbar);
    }
    __syncthreads();
    if (pfail || i < j || i >= nb) return;
    dd_t *d = A + (c0 + i) + lda * (long)(c0 + j);
    dd_t x = ld_dd(d);
    for (int k = 0; k < nbp; ++k) {
        const double2 pj = pre_sp[k * w + j], pi = pre_sp[k * w + i];
        x = dd_sub(x, dd_mul(dd_make(pj.x, pj.y), dd_make(pi.x, pi.y)));
    }
    st_dd(d, x);
}

static void panel_attr() {
    CK(cudaFuncSetAttribute(potrf_panel_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL_SMEM));
    CK(cudaFuncSetAttribute(potrf_panel_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL_SMEM));
}
// `below` rows of each of `count` matrices.  Few rows: 16 lanes a row keep a
// step's chain short; more rows than fill the SM sub-partitions (two rows a
// warp): 8 lanes, whose slots idle less.  1000 rows 14.3 us with 16, 15.6 with
// 8; 1500 rows 16.9 and 15.8.
constexpr long PANEL_FEW_ROWS = 1184;
static void panel_launch(cudaStream_t st, dd_t *A, long lda, int n, int c0, int below, int count, int *info, const dd_t *rdiag, const PotrfItem *list) {
    const long rows = (long)below * count;
    auto grid = [&](int c) { return dim3((unsigned)ceil_div(below, panel_rows(c)), (unsigned)count); };
    if (rows <= PANEL_FEW_ROWS) potrf_panel_kernel<16><<<grid(16), PANEL_THREADS, PANEL_SMEM, st>>>(A, lda, n, c0, info, rdiag, list);
    else potrf_panel_kernel<8><<<grid(8), PANEL_THREADS, PANEL_SMEM, st>>>(A, lda, n, c0, info, rdiag, list);
    CK_LAUNCH();
}

// Right-looking blocked Cholesky: per panel of POTRF_NB columns, factor the
// diagonal block, solve the rows below, then subtract the panel's outer
// product from the trailing lower triangle (GEMM_SUB keeps each entry's
// k-order).  info is a device int; 0 on success, else the failing column.
void potrf(cudaStream_t st, dd_t *A, long lda, int n, int *info_dev, dd_t *rdiag_dev, OzakiWork *tc) {
    if (n <= 0) return;
    static thread_local bool attr[64] = {};
    const int nbmax = POTRF_NB;
    const size_t smem_diag = sizeof(double2) * nbmax * nbmax;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (!attr[dev & 63]) {
        CK(cudaFuncSetAttribute(potrf_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_diag));
        panel_attr();
        CK(cudaFuncSetAttribute(potrf_diag_pre_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(double2) * nbmax * nbmax)));
        attr[dev & 63] = true;
    }
    if (tc && tc->side && n > 2 * nbmax) {
        // Split form with one block of lookahead: after panel k, the next
        // diagonal block takes panel k's update in dd (a small kernel) and
        // is factored on the side stream, on an SM the trailing update
        // leaves free, while the trailing update of panel k (all but that
        // block) runs; panel k+1 waits for both.
        {
            PROF_SCOPE("potrf_diag", st);
            potrf_diag_kernel<<<1, DIAG_THREADS, sizeof(double2) * nbmax * nbmax, st>>>(A, lda, nbmax, 0, info_dev, rdiag_dev, 0);
            CK_LAUNCH();
        }
        for (int c0 = 0;; c0 += nbmax) {
            const int nb = std::min(nbmax, n - c0);
            const int below = n - c0 - nb;
            if (below <= 0) break;
            {
                PROF_SCOPE("potrf_panel", st);
                panel_launch(st, A, lda, n, c0, below, 1, info_dev, rdiag_dev, nullptr);
            }
            const int c1 = c0 + nb, nb1 = std::min(nbmax, n - c1);
            {
                PROF_SCOPE("potrf_diag_pre", st);
                potrf_diag_pre_kernel<<<nb1, nbmax, sizeof(double2) * nbmax * nb, st>>>(A, lda, c1, nb1, nb, info_dev);
                CK_LAUNCH();
            }
            CK(cudaEventRecord(tc->ev_pre, st));
            CK(cudaStreamWaitEvent(tc->side, tc->ev_pre, 0));
            {
                PROF_SCOPE("potrf_diag", tc->side);
                potrf_diag_kernel<<<1, DIAG_THREADS, sizeof(double2) * nb1 * nb1, tc->side>>>(A, lda, nb1, c1, info_dev, rdiag_dev, 0);
                CK_LAUNCH();
            }
            CK(cudaEventRecord(tc->ev_diag, tc->side));
            if (below > nb1) {
                PROF_SCOPE("potrf_trailing_update_tc", st);
                ozaki_syrk_sub_lower(st, A + c1 + lda * (long)c0, lda, below, nb, A + c1 + lda * (long)c1, lda, *tc, nb1, 1);
            }
            CK(cudaStreamWaitEvent(st, tc->ev_diag, 0));
        }
        return;
    }
    for (int c0 = 0; c0 < n; c0 += nbmax) {
        const int nb = std::min(nbmax, n - c0);
        {
            PROF_SCOPE("potrf_diag", st);
            potrf_diag_kernel<<<1, DIAG_THREADS, sizeof(double2) * nb * nb, st>>>(A, lda, nb, c0, info_dev, rdiag_dev, 0);
            CK_LAUNCH();
        }
        const int below = n - c0 - nb;
        if (below <= 0) break;
        {
            PROF_SCOPE("potrf_panel", st);
            panel_launch(st, A, lda, n, c0, below, 1, info_dev, rdiag_dev, nullptr);
        }
        dd_t *panel = A + (c0 + nb) + lda * (long)c0;
        dd_t *trail = A + (c0 + nb) + lda * (long)(c0 + nb);
        if (tc) {
            PROF_SCOPE("potrf_trailing_update_tc", st);
            ozaki_syrk_sub_lower(st, panel, lda, below, nb, trail, lda, *tc);
        } else {
            PROF_SCOPE("potrf_trailing_update", st);
            gemm(st, 'N', 'T', GEMM_SUB, below, below, nb, panel, lda, 0, panel, lda, 0, trail, lda, 0, 1, true);
        }
    }
}

int potrf_info_check(int info) {
    if (info < 0) throw Error(ERR_CUDA, "potrf: a wait for a diagonal block's columns in the panel or the lookahead update ran out");
    return info;
}

void potrf_batched(cudaStream_t st, dd_t *A, long lda, int n, long sA, int batch, int *info_dev) {
    if (n <= 0 || batch <= 0) return;
    if (n > POTRF_NB) throw Error(ERR_ARG, "potrf_batched: order above one diagonal block");
    const size_t smem = sizeof(double2) * n * n;
    CK(cudaFuncSetAttribute(potrf_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(double2) * POTRF_NB * POTRF_NB)));
    potrf_diag_kernel<<<batch, DIAG_THREADS, smem, st>>>(A, lda, n, 0, info_dev, nullptr, sA);
    CK_LAUNCH();
}

// The trailing update of every matrix of a list after the panel at c0, 16 x 16
// tiles of the lower triangle (grid row y: matrix y); every entry's k-order is
// gemm's.
template <bool PIPE>
__global__ void __launch_bounds__(T16_THREADS, T16_CTAS) potrf_update_list_kernel(const PotrfItem *list, int c0) {
    __shared__ Tile16 S;
    const PotrfItem &it = list[blockIdx.y];
    const int c1 = c0 + POTRF_NB, w = it.n - c1;
    if (w <= 0 || *it.info != 0) return;
    const int t = blockIdx.x;
    int ti = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (ti * (ti + 1) / 2 > t) --ti;
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int i0 = ti * T16, j0 = (t - ti * (ti + 1) / 2) * T16;
    if (i0 >= w) return;
    const long lda = it.n;
    const dd_t *P = it.A + c1 + lda * c0;
    dd_t *C = it.A + c1 + lda * c1;
    const int gj = j0 + threadIdx.x % T16, gi = i0 + threadIdx.x / T16;
    dd_t acc[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) acc[r] = gi + 8 * r < w && gj < w ? ld_dd(C + gi + 8 * r + lda * gj) : dd_zero();
    tile16_sum<false, false, true, PIPE>(
        S, POTRF_NB, [&](int i, long k) { return i0 + i < w ? *reinterpret_cast<const double2 *>(P + i0 + i + lda * k) : make_double2(0.0, 0.0); },
        [&](int j, long k) { return j0 + j < w ? *reinterpret_cast<const double2 *>(P + j0 + j + lda * k) : make_double2(0.0, 0.0); }, acc);
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (gi + 8 * r < w && gi + 8 * r >= gj) st_dd(C + gi + 8 * r + lda * gj, acc[r]);
}

// Every matrix of a list: the block steps of potrf, each one launch over all
// matrices.  A batch of 16 problems (orders up to a few hundred): 0.4 ms a
// batch, launches included; column by column in global memory, one CTA a
// matrix, 1.07 ms.
void potrf_list(cudaStream_t st, const PotrfItem *list_dev, int count, int nmax) {
    if (count <= 0 || nmax <= 0) return;
    if (count > MAX_GRID_YZ) throw Error(ERR_ARG, "potrf_list: more matrices than a grid row holds");
    const size_t smem = sizeof(double2) * POTRF_NB * POTRF_NB;
    CK(cudaFuncSetAttribute(potrf_diag_list_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    panel_attr();
    for (int c0 = 0; c0 < nmax; c0 += POTRF_NB) {
        potrf_diag_list_kernel<<<count, DIAG_THREADS, smem, st>>>(list_dev, c0);
        CK_LAUNCH();
        const int below = nmax - c0 - POTRF_NB;
        if (below <= 0) break;
        panel_launch(st, nullptr, 0, 0, c0, below, count, nullptr, nullptr, list_dev);
        const long nt = ceil_div(below, T16), tiles = nt * (nt + 1) / 2;
        const dim3 grid((unsigned)tiles, count);
        if (tiles * count <= T16_PIPE_TILES)
            potrf_update_list_kernel<true><<<grid, T16_THREADS, 0, st>>>(list_dev, c0);
        else
            potrf_update_list_kernel<false><<<grid, T16_THREADS, 0, st>>>(list_dev, c0);
        CK_LAUNCH();
    }
}

// Zero the strict upper triangle (Lal::getCholesky, sdpa_linear.cpp:320-343).
__global__ void zero_upper_kernel(dd_t *A, long lda, int n, long sA) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)n * n) return;
    A += blockIdx.y * sA;
    int i = e % n, j = e / n;
    if (i < j) st_dd(A + i + lda * (long)j, dd_zero());
}
void zero_upper(cudaStream_t st, dd_t *A, long lda, int n, int batch, long sA) {
    if (n <= 0 || batch <= 0) return;
    if (batch > MAX_GRID_YZ) {
        for (int b0 = 0; b0 < batch; b0 += MAX_GRID_YZ) zero_upper(st, A + b0 * sA, lda, n, std::min(MAX_GRID_YZ, batch - b0), sA);
        return;
    }
    zero_upper_kernel<<<dim3(ceil_div((long)n * n, 256), batch), 256, 0, st>>>(A, lda, n, sA);
    CK_LAUNCH();
}

// ===================================================================== TRSV
// One cooperative launch per solve (or group of right-hand sides).  The
// matrix is cut into 64 x 64 tiles; CTA b owns the 64-entry blocks c = b, b +
// G, ... of x (forward) or the mirror order from the last block down
// (backward) and publishes each finished block through a per-block flag that
// holds the solve's epoch; right-hand side y is grid row y, with its own
// flags.  Each entry keeps the reference's own chain (mplapack/Rtrsv.cpp, the
// reference BLAS loop order):
//   "N": x(i) -= x(j) L(i,j) for j ascending (skipped when x(j) == 0),
//        then x(i) /= L(i,i) when x(i) != 0;
//   "T": t = x(j); t -= L(i,j) x(i) for i descending; x(j) = t / L(j,j).
// The time is that chain: per block its last tile's 64 dependent dd
// subtractions, then per entry a quotient, a product and a subtraction.  So
// all threads form a tile's products in place as soon as the block it
// multiplies is there, and two warps (an entry a lane) only subtract them,
// while the others bring the next tile; in the diagonal tile, warp 0 carries
// the chain x(t) -> x(t+1) in all lanes at once (no exchange in it), with the
// reciprocals of the diagonal formed beforehand (fastdiv.cuh), and updates the
// entries beyond beside it.
// A CTA waits for a block with an acquire load bounded by the solve's wait
// budget (2 s by default); on expiry it records the block in the error word
// and returns.  Tests of that path name a block whose flag is withheld.
// Measured, n = 1327: 402 us forward, 400 backward, for one right-hand side
// or two side by side (19 us a block, 13 of them in its diagonal tile); with
// one warp that multiplied, subtracted and divided for all 64 entries 747
// and 622 us each.
constexpr int TRSV_B = 64;
constexpr int TRSV_LD = 65;
constexpr int TRSV_THREADS = 256;
constexpr int TRSV_ONE_CTA = 8; // solves of at most 8 blocks (512 entries) run in one CTA
constexpr size_t TRSV_SMEM = 2 * sizeof(double2) * TRSV_B * TRSV_LD + 2 * sizeof(double2) * TRSV_B + sizeof(double) * TRSV_B;

struct TrsvArgs {
    const dd_t *L;
    long lda;
    int n, nblk, epoch;
    dd_t *x;
    long ldx;
    int *flags, *err; // nblk flags for each right-hand side
    unsigned long long wait_ns;
    int withhold; // a block whose flag is never published (-1: none)
};

__device__ __forceinline__ int ld_acquire_gpu(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int *p, int v) { asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Lane 0 of the calling warp waits until flags[blk] == epoch; every lane
// returns the outcome.
__device__ bool trsv_wait(const TrsvArgs &a, const int *flags, int blk) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        const unsigned long long t0 = global_ns();
        unsigned iter = 0;
        while (ld_acquire_gpu(flags + blk) != a.epoch) {
            if (ld_acquire_gpu(a.err) != 0 || ++iter > (1u << 26) || global_ns() - t0 > a.wait_ns) {
                atomicCAS(a.err, 0, blk + 1);
                ok = 0;
                break;
            }
            if (iter > 64) __nanosleep(64);
        }
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// T(i, j) = L(r0 + i, c0 + j) for i, j < 64 (zero outside the matrix).
// Every thread of [t0, t0 + nt) puts all its 16-byte copies in flight at
// once (cp.async; a source size of 0 writes zeros) and waits for them, so a
// tile costs one memory latency rather than one per element; the caller's
// __syncthreads then publishes the tile.
__device__ __forceinline__ void trsv_load_tile(double2 *T, const TrsvArgs &a, int r0, int c0, int t0, int nt) {
    for (int e = t0; e < TRSV_B * TRSV_B; e += nt) {
        const int i = e % TRSV_B, j = e / TRSV_B;
        const int gi = r0 + i, gj = c0 + j;
        const bool in = gi < a.n && gj < a.n;
        const dd_t *src = in ? a.L + gi + a.lda * (long)gj : a.L;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(T + i + TRSV_LD * j)), "l"(src),
                     "r"(in ? 16 : 0)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ dd_t ldcg_dd(const dd_t *p) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return dd_make(v.x, v.y);
}

// The diagonal tile by warp 0: entries lane and 32 + lane in v0, v1; steps s
// = 0 .. nb-1 (FWD) or nb-1 .. 0.  rd[t] = RN(1 / L(t,t).hi), or 0 where the
// quotient takes the plain form.
template <bool FWD> __device__ __forceinline__ void trsv_diag(const double2 *T, const double *rd, int nb, dd_t &v0, dd_t &v1) {
    const int lane = threadIdx.x & 31;
    // factor of entry e in step s
    auto el = [&](int e, int s) {
        const double2 v = FWD ? T[e + TRSV_LD * s] : T[s + TRSV_LD * e];
        return dd_make(v.x, v.y);
    };
    auto entry = [&](int e) { return shfl_dd(e < 32 ? v0 : v1, e & 31); };
    auto fast = [&](dd_t v, dd_t l, double y) { return dd_div_rest(v, l, div_corrected(v.hi, l.hi, y), y); };
    auto plain = [&](dd_t v, dd_t l) { return FWD && dd_is_zero(v) ? v : dd_div(v, l); };
    const int inc = FWD ? 1 : -1, first = FWD ? 0 : nb - 1, lastq = nb - 1;
    auto at = [&](int q) { return first + inc * min(q, lastq); };
    dd_t l = el(first, first), x = entry(first);
    x = rd[first] == 0.0 || !mid_range(x.hi) ? plain(x, l) : fast(x, l, rd[first]);
    // step q's operands, loaded a step ahead: the factors of the next entry
    // and of the lane's two, and the next diagonal; w: the next entry in
    // every lane, without step q's term
    int s = first, s1 = at(1);
    dd_t w = entry(s1), fn = el(s1, s), f0 = el(lane, s), f1 = el(32 + lane, s);
    double y = rd[s1];
    l = el(s1, s1);
    for (int q = 0; q < nb; ++q) {
        const int s2 = at(q + 2);
        const dd_t ln = el(s2, s2), gn = el(s2, s1), g0 = el(lane, s1), g1 = el(32 + lane, s1);
        const double yn = rd[s2];
        const bool skip = FWD && dd_is_zero(x);
        const dd_t nv = dd_sub(w, dd_mul(x, fn));
        const dd_t n0 = dd_sub(v0, dd_mul(x, f0)), n1 = dd_sub(v1, dd_mul(x, f1));
        if (!skip) w = nv;
        const bool u0 = !skip && (FWD ? lane > s && lane < nb : lane < s), u1 = !skip && (FWD ? 32 + lane > s && 32 + lane < nb : 32 + lane < s);
        v0 = lane == s ? x : u0 ? n0 : v0;
        v1 = 32 + lane == s ? x : u1 ? n1 : v1;
        x = fast(w, l, y);
        const dd_t wn = entry(s2);
        if (y == 0.0 || !mid_range(w.hi)) x = plain(w, l);
        w = wn, l = ln, fn = gn, f0 = g0, f1 = g1, y = yn;
        s = s1;
        s1 = s2;
    }
}

template <bool FWD> __global__ void __launch_bounds__(TRSV_THREADS) trsv_wave_kernel(TrsvArgs a) {
    extern __shared__ double2 trsv_sm[];
    double2 *xs = trsv_sm + 2 * TRSV_B * TRSV_LD, *vs = xs + TRSV_B;
    double *rd = reinterpret_cast<double *>(vs + TRSV_B);
    // zeros: the zero entries of the block's halves (forward: their steps are
    // skipped); two sets, since warps 0 and 1 read one while they subtract, each
    // at its own pace, and write the next block's before the next barrier
    __shared__ unsigned zeros[2][2];
    __shared__ int fail;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    dd_t *x = a.x + a.ldx * blockIdx.y;
    int *flags = a.flags + (long)a.nblk * blockIdx.y;
    if (tid == 0) fail = 0;
    // block c's tile with block p: rows c, columns p (FWD), or the transpose
    auto load = [&](int c, int p, int buf, int t0, int nt) {
        double2 *T = trsv_sm + buf * TRSV_B * TRSV_LD;
        trsv_load_tile(T, a, (FWD ? c : p) * TRSV_B, (FWD ? p : c) * TRSV_B, t0, nt);
    };
    for (int k = blockIdx.x; k < a.nblk; k += gridDim.x) {
        const int c = FWD ? k : a.nblk - 1 - k, r0 = c * TRSV_B, nb = min(TRSV_B, a.n - r0);
        dd_t v = dd_zero(); // thread t < 64: entry t
        if (tid < TRSV_B && r0 + tid < a.n) v = ld_dd(x + r0 + tid);
        if (tid < nb) {
            const double l = ld_dd(a.L + (r0 + tid) * (a.lda + 1)).hi;
            rd[tid] = mid_range(l) && !all_ones(l) ? __ddiv_rn(1.0, l) : 0.0;
        }
        load(c, FWD ? 0 : a.nblk - 1, 0, tid, TRSV_THREADS);
        for (int u = 0; u < k; ++u) {
            // the u-th block before c in the order of the terms
            const int p = FWD ? u : a.nblk - 1 - u, ib = min(TRSV_B, a.n - p * TRSV_B);
            double2 *T = trsv_sm + (u & 1) * TRSV_B * TRSV_LD;
            if (warp < 2) {
                if (!trsv_wait(a, flags, p)) {
                    if (lane == 0) fail = 1;
                } else {
                    const dd_t xa = tid < ib ? ldcg_dd(x + p * TRSV_B + tid) : dd_from(1.0);
                    xs[tid] = make_double2(xa.hi, xa.lo);
                    const unsigned z = __ballot_sync(0xffffffffu, FWD && dd_is_zero(xa));
                    if (lane == 0) zeros[u & 1][warp] = z;
                }
            }
            __syncthreads(); // the tile and block p are in
            if (fail) return;
            for (int e = tid; e < TRSV_B * TRSV_B; e += TRSV_THREADS) {
                const int i = e % TRSV_B, j = e / TRSV_B, t = FWD ? j : i;
                if (t >= ib) continue;
                double2 *at = T + i + TRSV_LD * j;
                const dd_t pr = dd_mul(dd_make(xs[t].x, xs[t].y), dd_make(at->x, at->y));
                *at = make_double2(pr.hi, pr.lo);
            }
            __syncthreads(); // its products are formed
            if (warp >= 2) {
                load(c, FWD ? p + 1 : p - 1, (u + 1) & 1, tid - 64, TRSV_THREADS - 64);
            } else {
                const double2 *at = FWD ? T + tid : T + TRSV_LD * tid;
                const int st = FWD ? TRSV_LD : 1;
                const unsigned zlo = zeros[u & 1][0], zhi = zeros[u & 1][1];
                if (ib == TRSV_B && (zlo | zhi) == 0u) {
                    double2 z[2][8]; // the next eight products come while these are subtracted
#pragma unroll
                    for (int q = 0; q < 8; ++q) z[0][q] = at[st * (FWD ? q : 63 - q)];
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (g < 7) z[(g + 1) & 1][q] = at[st * (FWD ? 8 * g + 8 + q : 55 - 8 * g - q)];
#pragma unroll
                        for (int q = 0; q < 8; ++q) v = dd_sub(v, dd_make(z[g & 1][q].x, z[g & 1][q].y));
                    }
                } else {
                    for (int q = 0; q < ib; ++q) {
                        const int t = FWD ? q : ib - 1 - q;
                        if ((t < 32 ? zlo : zhi) >> (t & 31) & 1u) continue;
                        v = dd_sub(v, dd_make(at[st * t].x, at[st * t].y));
                    }
                }
            }
        }
        if (tid < TRSV_B) vs[tid] = make_double2(v.hi, v.lo);
        __syncthreads(); // the diagonal tile is in
        if (warp == 0) {
            dd_t v0 = dd_make(vs[lane].x, vs[lane].y), v1 = dd_make(vs[32 + lane].x, vs[32 + lane].y);
            trsv_diag<FWD>(trsv_sm + (k & 1) * TRSV_B * TRSV_LD, rd, nb, v0, v1);
            if (r0 + lane < a.n) st_dd(x + r0 + lane, v0);
            if (r0 + 32 + lane < a.n) st_dd(x + r0 + 32 + lane, v1);
            __threadfence();
            __syncwarp();
            if (lane == 0 && c != a.withhold) st_release_gpu(flags + c, a.epoch);
        }
        __syncthreads();
    }
}

// Co-resident CTAs of a wave kernel on the current device.
static int trsv_grid_cap(const void *kernel) {
    int dev = 0, sms = 0, per = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRSV_SMEM));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, TRSV_THREADS, TRSV_SMEM));
    if (per < 1) throw Error(ERR_CUDA, "trsv: the wave kernel does not fit on an SM");
    return per * sms;
}

void trsv_lower(cudaStream_t st, char trans, const dd_t *L, long lda, int n, dd_t *x, TrsvSync &sync, bool shared_gpu, int nrhs, long ldx) {
    if (n <= 0 || nrhs <= 0) return;
    if (trans != 'N' && trans != 'T') throw Error(ERR_ARG, "trsv: trans must be 'N' or 'T'");
    const int nblk = ceil_div(n, TRSV_B);
    if ((long)nblk * nrhs > sync.capacity || !sync.flags) throw Error(ERR_ARG, "trsv: progress flags hold fewer blocks than the solve needs");
    PROF_SCOPE("trsv", st);
    if (++sync.epoch <= 0) sync.epoch = 1;
    TrsvArgs a{L, lda, n, nblk, sync.epoch, x, ldx, sync.flags, sync.flags + sync.capacity, sync.wait_ns, sync.withhold};
    const void *k = trans == 'N' ? (const void *)trsv_wave_kernel<true> : (const void *)trsv_wave_kernel<false>;
    static thread_local int cap[2][64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int &cp = cap[trans == 'N' ? 0 : 1][dev & 63];
    if (cp == 0) cp = trsv_grid_cap(k);
    if (nrhs > cp) throw Error(ERR_ARG, "trsv: more right-hand sides than the GPU holds CTAs");
    const int grid = std::min(nblk, cp / nrhs);
    if (shared_gpu && nblk <= TRSV_ONE_CTA) {
        // a short solve in one CTA, which walks the blocks in order and
        // never waits on another CTA: an ordinary launch, so it runs beside
        // other streams' work (a cooperative launch waits for room for its
        // whole grid); alone on the GPU the cooperative grid is faster
        if (trans == 'N')
            trsv_wave_kernel<true><<<dim3(1, nrhs), TRSV_THREADS, TRSV_SMEM, st>>>(a);
        else
            trsv_wave_kernel<false><<<dim3(1, nrhs), TRSV_THREADS, TRSV_SMEM, st>>>(a);
    } else {
        void *args[] = {&a};
        CK(cudaLaunchCooperativeKernel(k, dim3(grid, nrhs), TRSV_THREADS, args, TRSV_SMEM, st));
    }
    CK_LAUNCH();
}

void trsv_check(cudaStream_t st, const TrsvSync &sync) {
    if (!sync.flags) return;
    int err = 0;
    int *h = sync.h_err ? sync.h_err : &err;
    CK(cudaMemcpyAsync(h, sync.flags + sync.capacity, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (sync.wait_ev) {
        CK(cudaEventRecord(sync.wait_ev, st));
        CK(cudaEventSynchronize(sync.wait_ev));
    } else {
        CK(cudaStreamSynchronize(st));
    }
    err = *h;
    if (err != 0) {
        // clear the error word, so that the next solve starts afresh
        CK(cudaMemsetAsync(sync.flags + sync.capacity, 0, sizeof(int), st));
        CK(cudaStreamSynchronize(st));
    }
    if (err != 0)
        throw Error(ERR_CUDA, "trsv: a wait ran out of its " + std::to_string(sync.wait_ns / 1000000ull) + " ms budget for block " + std::to_string(err - 1) +
                                  " (solve abandoned)");
}

// ======================================================= triangular inverse
// X = inv(L): one CTA per column j, right-looking over k = j..n-1
// (Rtrsm "Left","Lower","N","N" on the identity).
__global__ void inv_lower_kernel(const dd_t *L, long lda, int n, dd_t *X, long ldx, long sL, long sX) {
    extern __shared__ double2 col[];
    const int j = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    L += blockIdx.y * sL;
    X += blockIdx.y * sX;
    for (int i = tid; i < n; i += nt) col[i] = make_double2(i == j ? 1.0 : 0.0, 0.0);
    __syncthreads();
    for (int k = j; k < n; ++k) {
        dd_t xk = dd_make(col[k].x, col[k].y);
        if (dd_is_zero(xk)) continue; // uniform across the CTA
        __syncthreads();
        if (tid == 0) {
            xk = dd_div(xk, ld_dd(L + k + lda * (long)k));
            col[k] = make_double2(xk.hi, xk.lo);
        }
        __syncthreads();
        xk = dd_make(col[k].x, col[k].y);
        for (int i = k + 1 + tid; i < n; i += nt) {
            dd_t v = dd_make(col[i].x, col[i].y);
            v = dd_sub(v, dd_mul(xk, ld_dd(L + i + lda * (long)k)));
            col[i] = make_double2(v.hi, v.lo);
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += nt) *reinterpret_cast<double2 *>(X + i + ldx * (long)j) = col[i];
}
// The same for n <= 2 blockDim: thread t holds rows t and t + blockDim; the
// L entries of step k+1 (its rows' L(i,k+1), and L(k+1,k+1) on thread 0)
// are loaded while step k runs, so no step waits on global memory.
constexpr int INV_THREADS = 128;
__global__ void __launch_bounds__(INV_THREADS) inv_lower_small_kernel(const dd_t *L, long lda, int n, dd_t *X, long ldx, long sL, long sX) {
    extern __shared__ double2 col[];
    const int j = blockIdx.x, tid = threadIdx.x;
    L += blockIdx.y * sL;
    X += blockIdx.y * sX;
    for (int i = tid; i < n; i += INV_THREADS) col[i] = make_double2(i == j ? 1.0 : 0.0, 0.0);
    auto lik_at = [&](int k, int r) {
        const int i = tid + INV_THREADS * r;
        return (i > k && i < n) ? ld_dd(L + i + lda * (long)k) : dd_zero();
    };
    dd_t lkk = tid == 0 ? ld_dd(L + j + lda * (long)j) : dd_zero();
    dd_t lik[2] = {lik_at(j, 0), lik_at(j, 1)};
    __syncthreads();
    for (int k = j; k < n; ++k) {
        const dd_t lkk_n = (tid == 0 && k + 1 < n) ? ld_dd(L + (k + 1) + lda * (long)(k + 1)) : dd_zero();
        const dd_t lik_n[2] = {lik_at(k + 1, 0), lik_at(k + 1, 1)};
        dd_t xk = dd_make(col[k].x, col[k].y);
        if (!dd_is_zero(xk)) { // uniform across the CTA
            if (tid == 0) {
                xk = dd_div(xk, lkk);
                col[k] = make_double2(xk.hi, xk.lo);
            }
            __syncthreads();
            xk = dd_make(col[k].x, col[k].y);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int i = tid + INV_THREADS * r;
                if (i > k && i < n) {
                    dd_t v = dd_make(col[i].x, col[i].y);
                    v = dd_sub(v, dd_mul(xk, lik[r]));
                    col[i] = make_double2(v.hi, v.lo);
                }
            }
            __syncthreads();
        }
        lkk = lkk_n;
        lik[0] = lik_n[0];
        lik[1] = lik_n[1];
    }
    for (int i = tid; i < n; i += INV_THREADS) *reinterpret_cast<double2 *>(X + i + ldx * (long)j) = col[i];
}

// The same for n <= 32 NW R with a column in registers: thread t holds rows j +
// t + 32 NW r.  A step's chain, a quotient (the reciprocals of the diagonal
// formed beforehand, fastdiv.cuh), a product and a subtraction, runs in every
// thread on the next entry, which the step before broadcast without its last
// term, so that the barrier of a step is not in the chain; L's entries are
// loaded two steps ahead.
// Measured, n = 500: 318 us; with the quotient on one thread between two
// barriers and L's column read when it is needed 540.  Up to 256 rows the form
// above is the faster one (n = 150: 36 us, this 46; n = 20: 7 and 10): its
// quotient costs one warp's issue slots, here every warp's.
template <int NW, int R>
__global__ void __launch_bounds__(32 * NW) inv_lower_rows_kernel(const dd_t *L, long lda, int n, dd_t *X, long ldx, long sL, long sX) {
    constexpr int T = 32 * NW;
    extern __shared__ double2 inv_sm[];
    double2 *dg = inv_sm, *sd = dg + n; // L(k,k), L(k+1,k)
    double *rc = reinterpret_cast<double *>(sd + n); // RN(1 / L(k,k).hi), or 0 where the quotient takes the plain form
    __shared__ double2 slot[2];
    const int j = blockIdx.x, tid = threadIdx.x;
    L += blockIdx.y * sL;
    X += blockIdx.y * sX;
    for (int i = j + tid; i < n; i += T) {
        const dd_t d = ld_dd(L + i + lda * (long)i);
        dg[i] = make_double2(d.hi, d.lo);
        rc[i] = mid_range(d.hi) && !all_ones(d.hi) ? __ddiv_rn(1.0, d.hi) : 0.0;
        if (i + 1 < n) sd[i] = *reinterpret_cast<const double2 *>(L + i + 1 + lda * (long)i);
    }
    auto load = [&](int k, dd_t *f) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = j + tid + T * r;
            f[r] = i > k && i < n ? ld_dd(L + i + lda * (long)k) : dd_zero(); // (i < n: k < n)
        }
    };
    dd_t v[R], fa[R], fb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = dd_from(tid + T * r == 0 ? 1.0 : 0.0);
    load(j, fa);
    load(j + 1, fb);
    __syncthreads();
    // entry k, and entry k+1 without step k's term, in every thread
    dd_t cur = dd_from(1.0), nxt = dd_zero();
    for (int k = j; k < n; ++k) {
        const dd_t l = dd_make(dg[k].x, dg[k].y), s = k + 1 < n ? dd_make(sd[k].x, sd[k].y) : dd_zero();
        const double y = rc[k];
        const bool zero = dd_is_zero(cur);
        dd_t x = dd_div_rest(cur, l, div_corrected(cur.hi, l.hi, y), y);
        if (y == 0.0 || !mid_range(cur.hi)) x = zero ? cur : dd_div(cur, l);
        const dd_t c = dd_sub(nxt, dd_mul(x, s));
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (j + T * r + T - 1 < k) continue; // rows above k
            const int i = j + tid + T * r;
            if (i == k) v[r] = x;
            if (i > k && !zero) v[r] = dd_sub(v[r], dd_mul(x, fa[r]));
            if (i == k + 2) slot[k & 1] = make_double2(v[r].hi, v[r].lo);
            fa[r] = fb[r];
        }
        load(k + 2, fb);
        __syncthreads();
        cur = zero ? nxt : c;
        nxt = dd_make(slot[k & 1].x, slot[k & 1].y); // (unused beyond the last row)
    }
    for (int i = tid; i < j; i += T) st_dd(X + i + ldx * (long)j, dd_zero());
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (j + tid + T * r < n) st_dd(X + j + tid + T * r + ldx * (long)j, v[r]);
}
template <int NW, int R> static void inv_rows_launch(cudaStream_t st, const dd_t *L, long lda, int n, dd_t *X, long ldx, int batch, long sL, long sX) {
    const size_t smem = (2 * sizeof(double2) + sizeof(double)) * n;
    inv_lower_rows_kernel<NW, R><<<dim3(n, batch), 32 * NW, smem, st>>>(L, lda, n, X, ldx, sL, sX);
    CK_LAUNCH();
}

void inv_lower(cudaStream_t st, const dd_t *L, long lda, int n, dd_t *X, long ldx, int batch, long sL, long sX) {
    if (n <= 0 || batch <= 0) return;
    if (batch > MAX_GRID_YZ) {
        for (int b0 = 0; b0 < batch; b0 += MAX_GRID_YZ) inv_lower(st, L + b0 * sL, lda, n, X + b0 * sX, ldx, std::min(MAX_GRID_YZ, batch - b0), sL, sX);
        return;
    }
    const size_t smem = sizeof(double2) * n;
    if (smem > 227 * 1024) throw Error(ERR_UNSUPPORTED, "inv_lower: block too large for one CTA");
    if (n <= 2 * INV_THREADS) {
        inv_lower_small_kernel<<<dim3(n, batch), INV_THREADS, smem, st>>>(L, lda, n, X, ldx, sL, sX);
        CK_LAUNCH();
        return;
    }
    if (n <= 512) return inv_rows_launch<4, 4>(st, L, lda, n, X, ldx, batch, sL, sX);
    if (n <= 1024) return inv_rows_launch<4, 8>(st, L, lda, n, X, ldx, batch, sL, sX);
    if (smem > 48 * 1024) CK(cudaFuncSetAttribute(inv_lower_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    inv_lower_kernel<<<dim3(n, batch), 128, smem, st>>>(L, lda, n, X, ldx, sL, sX);
    CK_LAUNCH();
}

// B = M^T M for lower M, entry by entry as Rtrmm("L","L","T","N") does in
// place: t = M(i,j) M(i,i); t += M(k,i) M(k,j), k = i+1..n-1 (terms with
// M(k,j) = 0, k < j, add exact zeros and are skipped).
__global__ void trmm_lt_kernel(const dd_t *M, long ldm, int n, dd_t *B, long ldb, long sM, long sB) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)n * n) return;
    M += blockIdx.y * sM;
    B += blockIdx.y * sB;
    int i = e % n, j = e / n;
    dd_t t = dd_mul(ld_dd(M + i + ldm * (long)j), ld_dd(M + i + ldm * (long)i));
    for (int k = max(i + 1, j); k < n; ++k) t = dd_acc(t, dd_mul(ld_dd(M + k + ldm * (long)i), ld_dd(M + k + ldm * (long)j)));
    st_dd(B + i + ldb * (long)j, t);
}
void trmm_lt(cudaStream_t st, const dd_t *M, long ldm, int n, dd_t *B, long ldb, int batch, long sM, long sB) {
    if (n <= 0 || batch <= 0) return;
    if (batch > MAX_GRID_YZ) {
        for (int b0 = 0; b0 < batch; b0 += MAX_GRID_YZ) trmm_lt(st, M + b0 * sM, ldm, n, B + b0 * sB, ldb, std::min(MAX_GRID_YZ, batch - b0), sM, sB);
        return;
    }
    trmm_lt_kernel<<<dim3(ceil_div((long)n * n, 128), batch), 128, 0, st>>>(M, ldm, n, B, ldb, sM, sB);
    CK_LAUNCH();
}

// =============================================================== symmetrize
__global__ void symmetrize_kernel(dd_t *A, int n, long sA) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)n * n) return;
    A += blockIdx.y * sA;
    int i = e % n, c = e / n;
    if (i <= c) return;
    dd_t v = dd_acc(ld_dd(A + i + (long)n * c), ld_dd(A + c + (long)n * i));
    v = dd_mul(dd_from(0.5), v);
    st_dd(A + i + (long)n * c, v);
    st_dd(A + c + (long)n * i, v);
}
void symmetrize(cudaStream_t st, dd_t *A, int n, int batch, long sA) {
    if (n <= 1 || batch <= 0) return;
    if (batch > MAX_GRID_YZ) {
        for (int b0 = 0; b0 < batch; b0 += MAX_GRID_YZ) symmetrize(st, A + b0 * sA, n, std::min(MAX_GRID_YZ, batch - b0), sA);
        return;
    }
    symmetrize_kernel<<<dim3(ceil_div((long)n * n, 256), batch), 256, 0, st>>>(A, n, sA);
    CK_LAUNCH();
}

// ================================================================ vector ops
__global__ void fill_kernel(dd_t *x, long n, dd_t v) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e < n) st_dd(x + e, v);
}
void fill(cudaStream_t st, dd_t *x, long n, dd_t v) {
    if (n <= 0) return;
    fill_kernel<<<ceil_div(n, 256), 256, 0, st>>>(x, n, v);
    CK_LAUNCH();
}

// y = a * y (Rscal: da * dx)
__global__ void scal_kernel(dd_t *y, long n, dd_t a) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e < n) st_dd(y + e, dd_mul(a, ld_dd(y + e)));
}
void scal(cudaStream_t st, dd_t *y, long n, dd_t a) {
    if (n <= 0) return;
    scal_kernel<<<ceil_div(n, 256), 256, 0, st>>>(y, n, a);
    CK_LAUNCH();
}

// y = x * a (Rcopy then Rscal)
__global__ void copy_scal_kernel(const dd_t *x, dd_t *y, long n, dd_t a) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e < n) st_dd(y + e, dd_mul(a, ld_dd(x + e)));
}
void copy_scal(cudaStream_t st, const dd_t *x, dd_t *y, long n, dd_t a) {
    if (n <= 0) return;
    copy_scal_kernel<<<ceil_div(n, 256), 256, 0, st>>>(x, y, n, a);
    CK_LAUNCH();
}

// z = x; z += a * y (Rcopy then Raxpy; Raxpy returns early when a == 0)
__global__ void axpy_kernel(const dd_t *x, const dd_t *y, dd_t *z, long n, dd_t a) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e < n) st_dd(z + e, dd_acc(ld_dd(x + e), dd_mul(a, ld_dd(y + e))));
}
void axpy(cudaStream_t st, const dd_t *x, const dd_t *y, dd_t *z, long n, dd_t a) {
    if (n <= 0) return;
    if (dd_is_zero(a)) {
        if (x != z) CK(cudaMemcpyAsync(z, x, sizeof(dd_t) * n, cudaMemcpyDeviceToDevice, st));
        return;
    }
    axpy_kernel<<<ceil_div(n, 256), 256, 0, st>>>(x, y, z, n, a);
    CK_LAUNCH();
}

// ================================================================ reductions
// Deterministic dd dot product.  Up to DOT_SEQ terms: one sequential chain,
// identical to Rdot with one OpenMP thread.  Longer: contiguous chunks summed
// sequentially, then a fixed pairwise tree (same result on every run).
constexpr int DOT_SEQ = 1024;
constexpr int DOT_THREADS = 256;

__global__ void __launch_bounds__(CHAIN_THREADS) dot_seq_kernel(const dd_t *x, long incx, const dd_t *y, long incy, long n, dd_t *out) {
    __shared__ double2 buf[2][CHAIN_CHUNK];
    const dd_t t = cta_chain(n, [&](long i) { return dd_mul(ld_dd(x + i * incx), ld_dd(y + i * incy)); }, buf);
    if (threadIdx.x == 0) st_dd(out, dd_acc(dd_zero(), t));
}

// Chains of a batch of equal-length dot products: CTA b, x + b sx, y + b
// sy, result out[b].
__global__ void __launch_bounds__(CHAIN_THREADS) dot_seq_batch_kernel(const dd_t *x, long sx, const dd_t *y, long sy, long n, dd_t *out) {
    __shared__ double2 buf[2][CHAIN_CHUNK];
    x += blockIdx.x * sx;
    y += blockIdx.x * sy;
    const dd_t t = cta_chain(n, [&](long i) { return dd_mul(ld_dd(x + i), ld_dd(y + i)); }, buf);
    if (threadIdx.x == 0) st_dd(out + blockIdx.x, dd_acc(dd_zero(), t));
}

__device__ dd_t block_tree(dd_t v, double2 *sh) {
    const int tid = threadIdx.x;
    sh[tid] = make_double2(v.hi, v.lo);
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (tid < s) {
            dd_t a = dd_make(sh[tid].x, sh[tid].y), b = dd_make(sh[tid + s].x, sh[tid + s].y);
            dd_t r = dd_add(a, b);
            sh[tid] = make_double2(r.hi, r.lo);
        }
        __syncthreads();
    }
    return dd_make(sh[0].x, sh[0].y);
}

__global__ void dot_chunk_kernel(const dd_t *x, long incx, const dd_t *y, long incy, long n, dd_t *partial) {
    __shared__ double2 sh[DOT_THREADS];
    const long nthr = (long)gridDim.x * DOT_THREADS;
    const long g = blockIdx.x * (long)DOT_THREADS + threadIdx.x;
    const long q = n / nthr, r = n % nthr;
    const long lo = g * q + min(g, r), hi = lo + q + (g < r ? 1 : 0);
    dd_t t = dd_zero();
    for (long i = lo; i < hi; ++i) t = dd_acc(t, dd_mul(ld_dd(x + i * incx), ld_dd(y + i * incy)));
    dd_t s = block_tree(t, sh);
    if (threadIdx.x == 0) st_dd(partial + blockIdx.x, s);
}
__global__ void tree_final_kernel(const dd_t *partial, int np, dd_t *out) {
    __shared__ double2 sh[DOT_THREADS];
    dd_t v = threadIdx.x < np ? ld_dd(partial + threadIdx.x) : dd_zero();
    dd_t s = block_tree(v, sh);
    if (threadIdx.x == 0) st_dd(out, s);
}

void dot(cudaStream_t st, const dd_t *x, long incx, const dd_t *y, long incy, long n, dd_t *out, dd_t *scratch) {
    if (n <= DOT_SEQ) {
        dot_seq_kernel<<<1, CHAIN_THREADS, 0, st>>>(x, incx, y, incy, n, out);
        CK_LAUNCH();
        return;
    }
    int nb = (int)std::min<long>(DOT_THREADS, ceil_div(n, 16L * DOT_THREADS));
    dot_chunk_kernel<<<nb, DOT_THREADS, 0, st>>>(x, incx, y, incy, n, scratch);
    CK_LAUNCH();
    tree_final_kernel<<<1, DOT_THREADS, 0, st>>>(scratch, nb, out);
    CK_LAUNCH();
}

void dot_batched(cudaStream_t st, const dd_t *x, long sx, const dd_t *y, long sy, long n, int batch, dd_t *out, dd_t *scratch) {
    if (batch <= 0) return;
    if (n <= DOT_SEQ) {
        dot_seq_batch_kernel<<<batch, CHAIN_THREADS, 0, st>>>(x, sx, y, sy, n, out);
        CK_LAUNCH();
        return;
    }
    for (int b = 0; b < batch; ++b) dot(st, x + b * sx, 1, y + b * sy, 1, n, out + b, scratch + 256 * (b % 8));
}

// max |x_i| (Residuals::computeMaxNorm) - exact in any order.
__global__ void maxabs_kernel(const dd_t *x, long n, dd_t *partial) {
    __shared__ double2 sh[DOT_THREADS];
    dd_t m = dd_zero();
    for (long i = blockIdx.x * (long)DOT_THREADS + threadIdx.x; i < n; i += (long)gridDim.x * DOT_THREADS) m = dd_max(m, dd_abs(ld_dd(x + i)));
    sh[threadIdx.x] = make_double2(m.hi, m.lo);
    __syncthreads();
    for (int s = DOT_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            dd_t a = dd_make(sh[threadIdx.x].x, sh[threadIdx.x].y), b = dd_make(sh[threadIdx.x + s].x, sh[threadIdx.x + s].y);
            dd_t r = dd_max(a, b);
            sh[threadIdx.x] = make_double2(r.hi, r.lo);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = dd_make(sh[0].x, sh[0].y);
}
__global__ void max_final_kernel(const dd_t *partial, int np, dd_t *out) {
    __shared__ double2 sh[DOT_THREADS];
    if (threadIdx.x < np) {
        const dd_t v = ld_dd(partial + threadIdx.x);
        sh[threadIdx.x] = make_double2(v.hi, v.lo);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    dd_t m = dd_zero();
    for (int i = 0; i < np; ++i) m = dd_max(m, dd_make(sh[i].x, sh[i].y));
    *out = m;
}
void maxabs(cudaStream_t st, const dd_t *x, long n, dd_t *out, dd_t *scratch) {
    int nb = (int)std::min<long>(DOT_THREADS, std::max(1u, ceil_div(n, 4L * DOT_THREADS)));
    maxabs_kernel<<<nb, DOT_THREADS, 0, st>>>(x, n, scratch);
    CK_LAUNCH();
    max_final_kernel<<<1, DOT_THREADS, 0, st>>>(scratch, nb, out);
    CK_LAUNCH();
}

} // namespace sddd
