// The device side of the reference's Newton step, update and residuals
// (sdpa_newton.cpp, sdpa_dataset.cpp), on block spaces resident in HBM.
#include "newton.h"

#include <algorithm>
#include <cstring>

#include "blas.h"
#include "devops.cuh"
#include "sparse_chol.h"

namespace sddd {

static const dd_t ONE = {1.0, 0.0};
static const dd_t MONE = {-1.0, 0.0};

// --------------------------------------------------- per-constraint A_k . M
// InputData::multi_InnerProductToA (sdpa_dataset.cpp:477-485) followed by
// "v = v * (-1); v = v + w" (the callers' Lal::let pair, Rscal then Raxpy).
//
// The product of a dense constraint matrix with a block of M is one chain of
// n^2 dd sums (Rdot's order), so a kernel can do no better than that chain's
// latency, 8 dependent FP64 operations (63 cycles) a term, and has to keep
// everything else off it.  inner_pairs_kernel gives a CTA up to 32 matrices
// of one block, one a lane of warp 0, which only adds: warp 1 brings the
// chunk of 32 terms of every matrix after next (cp.async, 512 contiguous
// bytes an instruction), warps 2 and 3 form the products of the next chunk
// (a term at a lane; rows are 33 entries apart, so that warp 0 reads them
// without bank conflicts).  Sparse matrices with long sums go through it
// too, one a CTA, the terms formed by all threads.  Then one thread a
// constraint adds its blocks' products in block order, short sparse products
// formed on the spot.
// Blocks 100 + 50, m = 1326: 0.40 ms; with the products formed by the adding
// warp 0.49 ms (the multiplications delay the chain in the FP64 pipe); one
// thread a constraint that streamed its matrices from global memory, block
// after block, took 2.24 ms.
constexpr int IP_CHUNK = 32, IP_LD = IP_CHUNK + 1, IP_THREADS = 128;
constexpr size_t IP_SMEM = sizeof(double2) * (4 * 32 * IP_LD + 2 * IP_CHUNK); // raw and product stages, M

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__global__ void __launch_bounds__(IP_THREADS) inner_pairs_kernel(const InnerTask *tasks, const int *pair_t, const int *pair_at,
                                                                const BlockView *views, const long *off, const dd_t *M, dd_t *prod) {
    extern __shared__ double2 ip_sm[];
    const InnerTask task = tasks[blockIdx.x];
    const BlockView &v = views[task.block];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = v.n;
    const dd_t *Ml = M + off[task.block];
    if (task.count < 0) {
        // one sparse matrix
        const int t = pair_t[task.first], o = v.coo_off[t], nnz = v.nnz[t], steps = sparse_dot_steps(nnz);
        const int *row = v.row + o, *col = v.col + o;
        const dd_t *val = v.val + o;
        constexpr int BUF = 4 * 32 * IP_LD;
        dd_t r = dd_zero();
        for (int base = 0; base < steps; base += BUF) {
            const int len = min(BUF, steps - base);
            for (int e = tid; e < len; e += IP_THREADS) {
                const dd_t x = sparse_dot_step(n, nnz, row, col, val, Ml, base + e);
                ip_sm[e] = make_double2(x.hi, x.lo);
            }
            __syncthreads();
            if (tid == 0)
                for (int e = 0; e < len; ++e) r = dd_acc(r, dd_make(ip_sm[e].x, ip_sm[e].y));
            __syncthreads();
        }
        if (tid == 0) st_dd(prod + pair_at[task.first], r);
        return;
    }
    const long nn = (long)n * n;
    const dd_t *A = v.dense + v.dense_off[pair_t[task.first + min(lane, task.count - 1)]];
    double2 *raw = ip_sm, *prd = ip_sm + 2 * 32 * IP_LD, *Ms = ip_sm + 4 * 32 * IP_LD;
    auto load = [&](long k0, int stage) { // warp 1
        if (k0 + lane < nn) cp_async16(Ms + stage * IP_CHUNK + lane, Ml + k0 + lane);
        for (int r = 0; r < task.count; ++r) {
            const dd_t *row = reinterpret_cast<const dd_t *>(__shfl_sync(0xffffffffu, (unsigned long long)A, r));
            if (k0 + lane < nn) cp_async16(raw + (stage * 32 + r) * IP_LD + lane, row + k0 + lane);
        }
        cp_async_commit();
    };
    auto form = [&](int stage) { // warps 2 and 3; terms past nn are never added
        const double2 y = Ms[stage * IP_CHUNK + lane];
        for (int r = warp - 2; r < task.count; r += 2) {
            const int at = (stage * 32 + r) * IP_LD + lane;
            const double2 x = raw[at];
            const dd_t q = dd_mul(dd_make(x.x, x.y), dd_make(y.x, y.y));
            prd[at] = make_double2(q.hi, q.lo);
        }
    };
    if (warp == 1) {
        load(0, 0);
        cp_async_wait<0>();
    }
    __syncthreads();
    if (warp == 1 && IP_CHUNK < nn) load(IP_CHUNK, 1);
    if (warp >= 2) form(0);
    dd_t t = dd_zero();
    int stage = 0;
    for (long k0 = 0; k0 < nn; k0 += IP_CHUNK, stage ^= 1) {
        if (warp == 1) cp_async_wait<0>();
        __syncthreads();
        if (warp > 0) {
            // chunk k0's products are formed; its raw stage is free
            if (warp == 1 && k0 + 2 * IP_CHUNK < nn) load(k0 + 2 * IP_CHUNK, stage);
            if (warp >= 2 && k0 + IP_CHUNK < nn) form(stage ^ 1);
            continue;
        }
        const double2 *p = prd + (stage * 32 + min(lane, task.count - 1)) * IP_LD;
        if (nn - k0 >= IP_CHUNK) {
            double2 x[2][8]; // the next eight come while these are added
#pragma unroll
            for (int u = 0; u < 8; ++u) x[0][u] = p[u];
#pragma unroll
            for (int q = 0; q < IP_CHUNK / 8; ++q) {
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (q + 1 < IP_CHUNK / 8) x[(q + 1) & 1][u] = p[8 * (q + 1) + u];
#pragma unroll
                for (int u = 0; u < 8; ++u) t = dd_acc(t, dd_make(x[q & 1][u].x, x[q & 1][u].y));
            }
        } else {
            const int len = (int)(nn - k0);
            for (int k = 0; k < len; ++k) t = dd_acc(t, dd_make(p[k].x, p[k].y));
        }
    }
    if (warp == 0 && lane < task.count) st_dd(prod + pair_at[task.first + lane], dd_acc(dd_zero(), t));
}

__global__ void constraint_inner_kernel(int m, const BlockView *views, const long *off, const int *cb_ptr, const int *cb_block, const int *cb_t,
                                        const dd_t *M, const dd_t *prod, const dd_t *addv, dd_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    dd_t ret = dd_zero();
    for (int p = cb_ptr[i]; p < cb_ptr[i + 1]; ++p) {
        const int l = cb_block[p], t = cb_t[p]; // t < 0: formed by a task
        dd_t tmp;
        if (t < 0) {
            tmp = ld_dd(prod + p);
        } else {
            const BlockView &v = views[l];
            const int o = v.coo_off[t];
            tmp = sparse_dot_dense(v.n, v.nnz[t], v.row + o, v.col + o, v.val + o, M + off[l]);
        }
        ret = dd_acc(ret, tmp);
    }
    st_dd(out + i, dd_acc(dd_mul(MONE, ret), dd_mul(ONE, ld_dd(addv + i))));
}

void constraint_inner(Context &c, const Space &M, const dd_t *addv, dd_t *out) {
    if (c.n_inner_tasks > 0) {
        static thread_local bool attr[64] = {};
        int dev = 0;
        CK(cudaGetDevice(&dev));
        if (!attr[dev & 63]) {
            CK(cudaFuncSetAttribute(inner_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IP_SMEM));
            attr[dev & 63] = true;
        }
        inner_pairs_kernel<<<c.n_inner_tasks, IP_THREADS, IP_SMEM, c.stream>>>(c.inner_tasks, c.inner_t, c.inner_at, c.views.p, c.d_off.p, M.buf.p,
                                                                      c.inner_prod());
        CK_LAUNCH();
    }
    constraint_inner_kernel<<<ceil_div(c.m, 64), 64, 0, c.stream>>>(c.m, c.views.p, c.d_off.p, c.cb_ptr.p, c.cb_block.p, c.cb_t.p, M.buf.p,
                                                                    c.inner_prod(), addv, out);
    CK_LAUNCH();
}

// ------------------------------------------------------- sum_k y_k A_k
// InputData::multi_plusToA (sdpa_dataset.cpp:488-493), entry by entry, then
// mode 0 (compute_DzMat, sdpa_newton.cpp:1318-1327): r = -r (+ D)
// mode 1 (Residuals::compute, sdpa_dataset.cpp:632-636): r = -r + C - Z
// One launch: CTA b takes the 128 entries of tasks[b] = (block, 128-chunk).
//
// Where every matrix of the block is dense, an entry's sum is a chain of dd
// multiply-adds over the constraints at 16 n^2 bytes a step, so a thread
// needs more loads in flight than the compiler keeps in registers: its terms
// come through a ring in shared memory, two stages of twelve terms, each
// thread copying and waiting for its own (cp.async), the y_k through a small
// ring a warp.  Bound by the chain, about 165 cycles a term with the product
// in it.  Blocks 100 + 50, m = 1326: 126 us; with eight loads ahead in
// registers and a launch a block 920 us; with the products formed by other
// warps, from registers, 180 us.  Stages of 8 terms, two or three: 145 us; of
// 16: 123 us, but slower where a block has few constraints.
constexpr int YA_THREADS = 128, YA_TERMS = 12, YA_STAGES = 2;
constexpr size_t YA_SMEM = sizeof(double2) * YA_STAGES * YA_TERMS * (YA_THREADS + YA_THREADS / 32);
static_assert(YA_TERMS <= 32, "a lane a y_k");
__global__ void __launch_bounds__(YA_THREADS) sum_yA_kernel(const BlockView *views, const int2 *tasks, const long *off, const dd_t *y, dd_t *out,
                                                           int mode, const dd_t *D, const dd_t *Z) {
    extern __shared__ double2 ya_sm[];
    const int2 task = tasks[blockIdx.x];
    const BlockView &v = views[task.x];
    const long ne = (long)v.n * v.n, base = off[task.x];
    const int tid = threadIdx.x, lane = tid & 31;
    const long e = (long)task.y * YA_THREADS + tid;
    dd_t acc = dd_zero();
    if (v.all_dense) {
        constexpr int RING = YA_STAGES * YA_TERMS;
        double2 *ring = ya_sm + tid, *yr = ya_sm + RING * YA_THREADS + (tid >> 5) * RING;
        const dd_t *A = v.dense + (e < ne ? e : ne - 1); // matrix t at t n^2
        const int *con = v.con, nc = v.nc;
        int k = lane < YA_TERMS && lane < nc ? con[lane] : 0; // of the next stage to go out
        auto issue = [&](int s) {
            const int t0 = s * YA_TERMS, slot = s % YA_STAGES * YA_TERMS;
#pragma unroll
            for (int u = 0; u < YA_TERMS; ++u)
                if (t0 + u < nc) cp_async16(ring + (slot + u) * YA_THREADS, A + (t0 + u) * ne);
            if (lane < YA_TERMS && t0 + lane < nc) {
                cp_async16(yr + slot + lane, y + k);
                if (t0 + YA_TERMS + lane < nc) k = con[t0 + YA_TERMS + lane];
            }
            cp_async_commit();
        };
#pragma unroll
        for (int s = 0; s < YA_STAGES - 1; ++s) issue(s);
        for (int s = 0; s * YA_TERMS < nc; ++s) {
            cp_async_wait<YA_STAGES - 2>();
            __syncwarp(); // the warp's y_k are in, and its stage s - 1 is read
            issue(s + YA_STAGES - 1);
            const int slot = s % YA_STAGES * YA_TERMS;
            auto term = [&](int u) {
                const double2 a = ring[(slot + u) * YA_THREADS], b = yr[slot + u];
                return dd_mul(dd_make(a.x, a.y), dd_make(b.x, b.y));
            };
            if ((s + 1) * YA_TERMS <= nc) {
#pragma unroll
                for (int u = 0; u < YA_TERMS; ++u) acc = dd_acc(acc, term(u));
            } else {
                for (int u = 0; s * YA_TERMS + u < nc; ++u) acc = dd_acc(acc, term(u));
            }
        }
        cp_async_wait<0>();
        if (e >= ne) return;
    } else {
        if (e >= ne) return;
        for (int q = v.el_ptr[e]; q < v.el_ptr[e + 1]; ++q) acc = dd_acc(acc, dd_mul(v.el_val[q], ld_dd(y + v.el_con[q])));
    }
    dd_t r = dd_mul(MONE, acc);
    if (mode == 0) {
        if (D) r = dd_acc(r, dd_mul(ONE, ld_dd(D + base + e)));
    } else {
        if (v.c_present) {
            if (v.c_dense) {
                r = dd_acc(r, dd_mul(ONE, ld_dd(v.c_dense_val + e)));
            } else {
                for (int q = v.c_el_ptr[e]; q < v.c_el_ptr[e + 1]; ++q) r = dd_acc(r, dd_mul(v.c_el_val[q], ONE));
            }
        }
        r = dd_acc(r, dd_mul(MONE, ld_dd(Z + base + e)));
    }
    st_dd(out + base + e, r);
}

void sum_yA(Context &c, const dd_t *y, Space &out, int mode, const Space *D, const Space *Z) {
    // the ring only where some block uses it
    size_t smem = 0;
    for (auto &b : c.blocks)
        if (b->all_dense && b->nc > 0) smem = YA_SMEM;
    static thread_local bool attr[64] = {};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (!attr[dev & 63]) {
        CK(cudaFuncSetAttribute(sum_yA_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)YA_SMEM));
        attr[dev & 63] = true;
    }
    sum_yA_kernel<<<c.n_yA_tasks, YA_THREADS, smem, c.stream>>>(c.views.p, c.yA_tasks, c.d_off.p, y, out.buf.p, mode, D ? D->buf.p : nullptr,
                                                               Z ? Z->buf.p : nullptr);
    CK_LAUNCH();
}

// ------------------------------------------------------------ init point
__global__ void set_identity_kernel(dd_t *A, int n, dd_t v) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)n * n) return;
    st_dd(A + e, (e % n == e / n) ? v : dd_zero());
}
static void set_identity(Context &c, Space &s, dd_t v) {
    for (int l = 0; l < c.nSDP; ++l) {
        int n = c.sizes[l];
        set_identity_kernel<<<ceil_div((long)n * n, 256), 256, 0, c.stream>>>(s.blk(c.off, l), n, v);
        CK_LAUNCH();
    }
}

void init_point(Context &c, dd_t lambda) {
    set_identity(c, c.X, lambda);
    set_identity(c, c.Z, lambda);
    fill(c.stream, c.y.p, c.m, dd_zero());
    dd_t ris = dd_div(ONE, dd_sqrt(lambda));
    set_identity(c, c.invCholX, ris);
    set_identity(c, c.invCholZ, ris);
    set_identity(c, c.invZ, dd_div(ONE, lambda));
}

// ------------------------------------------------------- inverses of X, Z
// Jal::getInvChol / getInvCholAndInv (sdpa_jordan.cpp:123-170): copy,
// Rpotrf, zero the upper triangle, Rtrsm on the identity; for Z also
// Z^-1 = L_Z^-T L_Z^-1 by Rtrmm.
void compute_inverse_async(Context &c) {
    cudaStream_t st = c.stream;
    if (!c.aux) {
        CK(cudaStreamCreateWithFlags(&c.aux, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&c.aux_fork, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&c.aux_join, cudaEventDisableTiming));
    }
    CK(cudaMemsetAsync(c.info.p, 0, sizeof(int) * 2, st));
    CK(cudaMemcpyAsync(c.W1.buf.p, c.X.buf.p, sizeof(dd_t) * c.space_len, cudaMemcpyDeviceToDevice, st));
    CK(cudaMemcpyAsync(c.W2.buf.p, c.Z.buf.p, sizeof(dd_t) * c.space_len, cudaMemcpyDeviceToDevice, st));
    // X's factors on the main stream, Z's (and Z^-1) on the second one
    CK(cudaEventRecord(c.aux_fork, st));
    CK(cudaStreamWaitEvent(c.aux, c.aux_fork, 0));
    for (int side = 0; side < 2; ++side) {
        cudaStream_t s = side == 0 ? st : c.aux;
        const Space &W = side == 0 ? c.W1 : c.W2;
        Space &inv = side == 0 ? c.invCholX : c.invCholZ;
        int *info = c.info.p + side;
        dd_t *rdiag = c.rdiag.p + 128 * side;
        for (const BlockRun &r : c.runs) {
            const int n = r.n;
            const long nn = (long)n * n;
            dd_t *w = W.blk(c.off, r.first);
            if (n <= POTRF_NB) {
                potrf_batched(s, w, n, n, nn, r.count, info);
            } else {
                for (int t = 0; t < r.count; ++t) potrf(s, w + t * nn, n, n, info, rdiag);
            }
            zero_upper(s, w, n, n, r.count, nn);
            inv_lower(s, w, n, n, inv.blk(c.off, r.first), n, r.count, nn, nn);
            if (side == 1) trmm_lt(s, c.invCholZ.blk(c.off, r.first), n, n, c.invZ.blk(c.off, r.first), n, r.count, nn, nn);
        }
    }
    CK(cudaEventRecord(c.aux_join, c.aux));
    CK(cudaStreamWaitEvent(st, c.aux_join, 0));
}

bool compute_inverse(Context &c) {
    compute_inverse_async(c);
    ScalarBatch sb(c);
    const int g = sb.inverse_info();
    sb.fetch();
    return sb.inverse_ok(g);
}

int ScalarBatch::inverse_info() {
    const int g = group(1);
    CK(cudaMemcpyAsync(c.scal.p + groups[g].first, c.info.p, 2 * sizeof(int), cudaMemcpyDeviceToDevice, c.stream));
    return g;
}

bool ScalarBatch::inverse_ok(int g) const {
    int info[2];
    std::memcpy(info, &host[groups[g].first], sizeof(info));
    potrf_info_check(info[0]);
    potrf_info_check(info[1]);
    return info[0] == 0 && info[1] == 0;
}

// ------------------------------------------------------------ Newton step
void triple(Context &c, const Space &A, const Space &B, const Space &C, Space &out) {
    // Jal::ns_jordan_triple_product: work = A B; out = work C (two Rgemm)
    for (const BlockRun &r : c.runs) {
        const int n = r.n, l = r.first;
        const long nn = (long)n * n;
        gemm(c.stream, 'N', 'N', GEMM_STORE, n, n, n, A.blk(c.off, l), n, nn, B.blk(c.off, l), n, nn, c.W2.blk(c.off, l), n, nn, r.count, false);
        gemm(c.stream, 'N', 'N', GEMM_STORE, n, n, n, c.W2.blk(c.off, l), n, nn, C.blk(c.off, l), n, nn, out.blk(c.off, l), n, nn, r.count, false);
    }
}

void make_rhs(Context &c, bool corrector, dd_t beta_mu, bool dual_infeasible) {
    cudaStream_t st = c.stream;
    const long L = c.space_len;
    // r_zinv = beta*mu * Z^-1 - X  (compute_rMat, sdpa_newton.cpp:821-837)
    copy_scal(st, c.invZ.buf.p, c.rzinv.buf.p, L, beta_mu);
    axpy(st, c.rzinv.buf.p, c.X.buf.p, c.rzinv.buf.p, L, MONE);
    if (corrector) {
        triple(c, c.Dx, c.Dz, c.invZ, c.W1);
        axpy(st, c.rzinv.buf.p, c.W1.buf.p, c.rzinv.buf.p, L, MONE);
    }
    // Make_gVec (sdpa_newton.cpp:839-893)
    if (dual_infeasible) {
        if (!corrector) triple(c, c.X, c.dualMat, c.invZ, c.xrdzinv);
        axpy(st, c.rzinv.buf.p, c.xrdzinv.buf.p, c.W1.buf.p, L, MONE);
    } else {
        CK(cudaMemcpyAsync(c.W1.buf.p, c.rzinv.buf.p, sizeof(dd_t) * L, cudaMemcpyDeviceToDevice, st));
    }
    constraint_inner(c, c.W1, c.primalVec.p, c.g.p);
}

int schur_factor(Context &c) {
    if (c.sparse_active()) {
        // Lal::getCholesky(SparseMatrix&, int*) reports no failure: a
        // negative pivot becomes a zero row (sdpa_linear.cpp:366-372)
        c.winv_valid = false;
        sparse_factor_B(c);
        return 0;
    }
    CK(cudaMemsetAsync(c.info.p, 0, sizeof(int), c.stream));
    OzakiWork *tc = c.tc_slices > 0 ? &tc_work(c, c.m, c.tc_slices) : nullptr;
    c.winv_valid = false;
    potrf(c.stream, c.B.p, c.m, c.m, c.info.p, c.rdiag.p, tc);
    int info = 0;
    d2h(c, &info, c.info.p, sizeof(int));
    potrf_info_check(info);
    if (tc) {
        ozaki_check(c.stream, *tc);
        if (info == 0) {
            // the split form's solves go by blocks (trsv_blocked)
            c.trsv_winv.alloc((size_t)ceil_div(c.m, 64) * 64 * 64);
            trsv_diag_inverse(c.stream, c.B.p, c.m, c.m, c.trsv_winv.p);
            c.winv_valid = true;
        }
    }
    return info;
}

void solve_B(Context &c, dd_t *x) {
    if (c.sparse_active()) {
        sparse_solve(c, x);
        return;
    }
    TrsvSync &sync = trsv_sync(c, c.m);
    if (c.winv_valid) {
        trsv_blocked(c.stream, 'N', c.B.p, c.m, c.m, c.trsv_winv.p, x, sync);
        trsv_blocked(c.stream, 'T', c.B.p, c.m, c.m, c.trsv_winv.p, x, sync);
    } else {
        trsv_lower(c.stream, 'N', c.B.p, c.m, c.m, x, sync, c.shared_gpu);
        trsv_lower(c.stream, 'T', c.B.p, c.m, c.m, x, sync, c.shared_gpu);
    }
    trsv_check(c.stream, sync);
}

void solve_dy(Context &c) {
    CK(cudaMemcpyAsync(c.Dy.p, c.g.p, sizeof(dd_t) * c.m, cudaMemcpyDeviceToDevice, c.stream));
    solve_B(c, c.Dy.p);
}

void make_dz_dx(Context &c, bool dual_infeasible) {
    sum_yA(c, c.Dy.p, c.Dz, 0, dual_infeasible ? &c.dualMat : nullptr, nullptr);
    triple(c, c.X, c.Dz, c.invZ, c.W1);
    axpy(c.stream, c.rzinv.buf.p, c.W1.buf.p, c.Dx.buf.p, c.space_len, MONE);
    for (const BlockRun &r : c.runs) symmetrize(c.stream, c.Dx.blk(c.off, r.first), r.n, r.count, (long)r.n * r.n);
}

// ------------------------------------------------------------ inner products
// Each reduction writes its partial results (one per block, or one) to
// slots of c.scal; a ScalarBatch lays several reductions side by side and
// reads them all back with one copy, so that independent scalars of one
// step cost one host round trip.  The host sums a group's slots in order
// from zero with "+=", as the reference sums its per-block results.
int ScalarBatch::group(int count) {
    groups.push_back({used, count});
    used += count;
    if ((size_t)used > c.scal.n) throw Error(ERR_STATE, "scalar batch: more result slots than the context holds");
    return (int)groups.size() - 1;
}

void ScalarBatch::fetch() {
    host.resize(used);
    if (used > 0) d2h(c, host.data(), c.scal.p, sizeof(dd_t) * used);
}

dd_t ScalarBatch::sum(int g) const {
    dd_t r = dd_zero();
    for (int s = 0; s < groups[g].second; ++s) r = dd_acc(r, host[groups[g].first + s]);
    return r;
}

dd_t ScalarBatch::value(int g) const { return host[groups[g].first]; }

// Lal::getInnerProduct(DenseLinearSpace, DenseLinearSpace)
// (sdpa_linear.cpp:1571-1611): Rdot per block, summed with "+=".
int ScalarBatch::inner_space(const Space &a, const Space &b) {
    const int g = group(c.nSDP);
    dd_t *out = c.scal.p + groups[g].first;
    for (const BlockRun &r : c.runs) {
        const long nn = (long)r.n * r.n;
        dot_batched(c.stream, a.blk(c.off, r.first), nn, b.blk(c.off, r.first), nn, nn, r.count, out + r.first, c.red.p);
    }
    return g;
}

// The blocks whose product with C is one chain (sparse C, or dense C of at
// most DOT_SEQ_TERMS entries) in one launch: CTA l, result to its slot.
constexpr long DOT_SEQ_TERMS = 1024; // the longest dot that dot() runs as one chain
__global__ void __launch_bounds__(CHAIN_THREADS) inner_C_small_kernel(const BlockView *views, const int *slot, const long *off, const dd_t *x,
                                                                    dd_t *out) {
    __shared__ double2 buf[2][CHAIN_CHUNK];
    const int l = blockIdx.x;
    const BlockView &v = views[l];
    const int s = slot[l];
    if (s < 0 || !v.c_present) return;
    const dd_t *D = x + off[l];
    dd_t r;
    if (!v.c_dense) {
        const int n = v.n, nnz = v.c_nnz, *row = v.c_row, *col = v.c_col;
        const dd_t *val = v.c_val;
        r = cta_chain(sparse_dot_steps(nnz), [&](long e) { return sparse_dot_step(n, nnz, row, col, val, D, (int)e); }, buf);
    } else {
        const long nn = (long)v.n * v.n;
        if (nn > DOT_SEQ_TERMS) return;
        const dd_t *C = v.c_dense_val;
        r = dd_acc(dd_zero(), cta_chain(nn, [&](long e) { return dd_mul(ld_dd(C + e), ld_dd(D + e)); }, buf));
    }
    if (threadIdx.x == 0) st_dd(out + s, r);
}

// Lal::getInnerProduct(SparseLinearSpace C, DenseLinearSpace X)
// (sdpa_linear.cpp:1616-1650) over C's nonzero SDP blocks: one result slot
// per such block, summed in block order on the host.
int ScalarBatch::inner_C(const Space &x) {
    if (c.c_slot_host.size() != (size_t)c.nSDP) {
        c.c_slot_host.assign(c.nSDP, -1);
        c.c_nslots = 0;
        for (int l = 0; l < c.nSDP; ++l)
            if (c.blocks[l]->c_present) c.c_slot_host[l] = c.c_nslots++;
        c.c_slot.upload(c.c_slot_host, c.stream);
    }
    const int g = group(c.c_nslots);
    if (c.c_nslots == 0) return g;
    dd_t *out = c.scal.p + groups[g].first;
    inner_C_small_kernel<<<c.nSDP, CHAIN_THREADS, 0, c.stream>>>(c.views.p, c.c_slot.p, c.d_off.p, x.buf.p, out);
    CK_LAUNCH();
    for (int l = 0; l < c.nSDP; ++l) {
        const BlockDev &bd = *c.blocks[l];
        const long nn = (long)bd.n * bd.n;
        if (bd.c_present && bd.c_dense && nn > DOT_SEQ_TERMS)
            dot(c.stream, bd.c_dense_val.p, 1, x.blk(c.off, l), 1, nn, out + c.c_slot_host[l], c.red.p + 256 * (c.c_slot_host[l] % 8));
    }
    return g;
}

// Lal::getInnerProduct(Vector, Vector): Rdot over m.
int ScalarBatch::inner_b(const dd_t *v) {
    const int g = group(1);
    dot(c.stream, c.b.p, 1, v, 1, c.m, c.scal.p + groups[g].first, c.red.p);
    return g;
}

// max |x_i| (Residuals::computeMaxNorm): one slot, taken as is.
int ScalarBatch::maxabs_of(const dd_t *x, long n, int scratch) {
    const int g = group(1);
    maxabs(c.stream, x, n, c.scal.p + groups[g].first, c.red.p + 512 * scratch);
    return g;
}

dd_t inner_space(Context &c, const Space &a, const Space &b) {
    ScalarBatch sb(c);
    const int g = sb.inner_space(a, b);
    sb.fetch();
    return sb.sum(g);
}

dd_t inner_C(Context &c, const Space &x) {
    ScalarBatch sb(c);
    const int g = sb.inner_C(x);
    sb.fetch();
    return sb.sum(g);
}

dd_t inner_b(Context &c, const dd_t *v) {
    ScalarBatch sb(c);
    const int g = sb.inner_b(v);
    sb.fetch();
    return sb.sum(g);
}

// ----------------------------------------------------------------- update
void update_point(Context &c, dd_t alphaP, dd_t alphaD) {
    axpy(c.stream, c.X.buf.p, c.Dx.buf.p, c.X.buf.p, c.space_len, alphaP);
    axpy(c.stream, c.y.p, c.Dy.p, c.y.p, c.m, alphaD);
    axpy(c.stream, c.Z.buf.p, c.Dz.buf.p, c.Z.buf.p, c.space_len, alphaD);
}

// -------------------------------------------------------------- residuals
// Residuals::compute (sdpa_dataset.cpp:625-645): the primal residual vector
// and the dual residual matrix, then their max-abs norms into the batch.
void ScalarBatch::residuals(int &gPrimal, int &gDual) {
    constraint_inner(c, c.X, c.b.p, c.primalVec.p);
    sum_yA(c, c.y.p, c.dualMat, 1, nullptr, &c.Z);
    gPrimal = maxabs_of(c.primalVec.p, c.m, 0);
    gDual = maxabs_of(c.dualMat.buf.p, c.space_len, 1);
}

void residuals(Context &c, dd_t &normPrimal, dd_t &normDual) {
    ScalarBatch sb(c);
    int gp, gd;
    sb.residuals(gp, gd);
    sb.fetch();
    normPrimal = sb.value(gp);
    normDual = sb.value(gd);
}

// sum_b sum_i S_b(i,i) lambda in order; dim[b]: rows before block b.
__global__ void __launch_bounds__(CHAIN_THREADS) lambda_trace_kernel(const dd_t *S, const long *off, const int *dim, int nb, double lambda, dd_t *out) {
    __shared__ double2 buf[2][CHAIN_CHUNK];
    const dd_t r = cta_chain(
        dim[nb],
        [&](long e) {
            int lo = 0, hi = nb; // the block with dim[lo] <= e < dim[lo + 1]
            while (hi - lo > 1) {
                const int mid = (lo + hi) / 2;
                if (dim[mid] <= e)
                    lo = mid;
                else
                    hi = mid;
            }
            const long i = e - dim[lo], n = dim[lo + 1] - dim[lo];
            return dd_mul_d(ld_dd(S + off[lo] + i + n * i), lambda);
        },
        buf);
    if (threadIdx.x == 0) st_dd(out, r);
}

int ScalarBatch::lambda_trace(const Space &s, double lambda) {
    const int g = group(1);
    lambda_trace_kernel<<<1, CHAIN_THREADS, 0, c.stream>>>(s.buf.p, c.d_off.p, c.d_dim, c.nSDP, lambda, c.scal.p + groups[g].first);
    CK_LAUNCH();
    return g;
}

dd_t lambda_trace(Context &c, const Space &s, double lambda) {
    ScalarBatch sb(c);
    const int g = sb.lambda_trace(s, lambda);
    sb.fetch();
    return sb.sum(g);
}

} // namespace sddd
