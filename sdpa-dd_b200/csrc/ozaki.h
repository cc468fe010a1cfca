// Tensor-core split of the Cholesky trailing update: C(lower) -= P P^T with
// dd operands cut into signed integer digits (an Ozaki-style
// error-free split) and multiplied on the INT8 tensor cores (tcgen05,
// kind::i8) with exact int32 accumulation, then rebuilt in dd.
#pragma once
#include "common.cuh"

namespace sddd {

constexpr int OZ_MAX_SLICES = 16; // 7-bit slices a caller may ask for
// Base-256 digits that carry `slices` 7-bit slices in the trailing update: one
// bit more than the slices have, since rows whose largest entry lies just below a
// power of two take a scale one bit larger than 7-bit digits need (ozaki.cu).
constexpr int ozaki_digits(int slices) { return (7 * slices + 1 + 7) / 8; }
constexpr int OZ_MAX_DIGITS = ozaki_digits(OZ_MAX_SLICES);
constexpr int OZ_K = 64;        // panel width the split handles (K of the update)
constexpr int OZ_ROWS_A = 128;  // output tile rows (MMA M)
constexpr int OZ_COLS_B = 16;   // output tile columns (per B digit)

// Device workspace of the split: digits for `row_cap` rows (a multiple of
// 128), row exponents and an error word.
struct OzakiWork {
    int8_t *digits = nullptr; // row_cap x OZ_MAX_DIGITS x 64 bytes by 16-row block: each block's digits contiguous
    int *exps = nullptr;      // row_cap
    int *err = nullptr;       // 0, or the code of a wait that gave up
    int *h_err = nullptr;     // pinned host word for reading err (or null)
    cudaEvent_t wait_ev = nullptr; // blocking-sync event to wait on (or null: stream sync)
    int row_cap = 0;
    int slices_used = 16;     // 7-bit slices per value (8..16)
    unsigned long long wait_ns = 2000000000ull; // budget of one mbarrier wait
    // the Cholesky's lookahead: the next diagonal block is factored on
    // `side` while the trailing update runs (ev_pre: its block is ready;
    // ev_diag: it is factored)
    cudaStream_t side = nullptr;
    cudaEvent_t ev_pre = nullptr, ev_diag = nullptr;
};

// C(i, j) -= sum_k P(i, k) P(j, k) for rows/cols < n with i >= j; P is
// n x k (k <= 64) column-major with leading dimension ldp, C n x n with ldc.
// Rows below `skip` (the leading skip x skip block, updated elsewhere) are
// left alone; `reserve_sms` SMs are left free for concurrent kernels.
void ozaki_syrk_sub_lower(cudaStream_t st, const dd_t *P, long ldp, int n, int k, dd_t *C, long ldc, OzakiWork &w, int skip = 0,
                          int reserve_sms = 0);
// Throws when a launch since the last check gave up waiting (synchronises st).
void ozaki_check(cudaStream_t st, const OzakiWork &w);

// The split of a long product C(i,j) = sum_k W(i,k) V(j,k), i >= j (the
// Schur complement's F1 pair products): W and V n x K, row r at
// W + r * ldw (K contiguous dd); C n x n column-major, lower triangle
// stored.  K <= OG_MAX_K (every diagonal of slice products accumulates
// exactly in int32 over the whole K).
constexpr long OG_MAX_K = 32767;
struct OzakiGemmWork {
    int8_t *sw = nullptr, *sv = nullptr; // slices of W and V
    size_t slice_bytes = 0;              // bytes of each slice buffer
    int *ew = nullptr, *ev = nullptr;    // row exponents (rows_cap each)
    int rows_cap = 0;
    int *err = nullptr;
    int *h_err = nullptr;
    cudaEvent_t wait_ev = nullptr;
    int slices = 16;
    unsigned long long wait_ns = 2000000000ull;
};
// Workspace bytes of one slice buffer for n rows, K values and S slices.
inline size_t ozaki_gemm_slice_bytes(int n, long K, int slices) {
    const long rows = (long)((n + 127) / 128) * 128, kpad = (K + 63) / 64 * 64;
    return (size_t)slices * rows * kpad;
}
void ozaki_gemm_lower(cudaStream_t st, const dd_t *W, long ldw, const dd_t *V, long ldv, int n, long K, dd_t *C, long ldc, OzakiGemmWork &w);
// Throws when a launch since the last check gave up waiting (synchronises st).
void ozaki_gemm_check(cudaStream_t st, const OzakiGemmWork &w);

} // namespace sddd
