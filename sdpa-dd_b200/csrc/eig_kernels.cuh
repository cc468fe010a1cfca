// Kernels of the step-length eigenvalue (eig.cu), declared for the other
// translation units that launch them on their own buffers.
#pragma once

#include "common.cuh"

namespace sddd {

constexpr int LZ_THREADS = 512; // threads of a CTA of the Lanczos kernel
constexpr int LZ_KMAX = 128;    // bound on the Lanczos steps held in shared memory
constexpr int LZ_WORK = 3;      // vectors of work a block may need in global memory

// One cluster per block id: lambda_min(L D L^T) of block ids[c] (order
// sizes[b], at most maxn, data at L/D + off[b]); with nsp = 2 clusters nb ..
// 2 nb - 1 take the same nb blocks of a second space (L2, D2).  work holds
// LZ_WORK maxn dd values per cluster at stride work_stride; the results go
// to out[c].
void launch_lanczos(cudaStream_t st, const int *ids, int nb, int nsp, long maxn, const int *sizes, const long *off, const dd_t *L, const dd_t *D,
                    const dd_t *L2, const dd_t *D2, dd_t *work, long work_stride, dd_t *out);

// One warp per block id: smallest eigenvalue of the lower triangle of the
// symmetric M (order <= 32) at Msp + off[b]; the result goes to out[blockIdx.x].
__global__ void __launch_bounds__(32) small_min_eig_kernel(const int *blk_ids, const int *sizes, const long *off, const dd_t *Msp, dd_t *out);

} // namespace sddd
