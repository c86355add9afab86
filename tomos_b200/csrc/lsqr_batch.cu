// lsqr_batch.cu -- K least-squares problems min ||A x_k - b_k|| over one A at
// once (tomos_lsqr_solve_batch_dense): one LSQR recurrence per column, the
// passes over A shared.
//
// One column's iteration is a pass over A and a few microseconds of n-side
// work, so K columns solved one after the other read A K times as often as
// they need to.  Here an iteration is one pass for all K columns
// (multi_rows_kernel) and one n-side launch, a cluster per column; columns
// whose cycle has ended idle until the last one's has.  The restart passes
// that certify a column run on their own, as in tomos_lsqr_solve_dense.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "gemv.cuh"
#include "lsqr.cuh"
#include "mbarrier.cuh"  // smem_addr

namespace tomos_b200 {

namespace {

// ut_k = cp_k A p_k + cu_k u_k and A^T ut_k for K <= 8 columns from one read
// of A (FP32, rows 16-byte aligned, n <= 512).  A CTA an SM streams tiles of
// 32 rows through two shared-memory buffers; of a tile in shared memory
//   dots    warp w takes rows 4 w .. 4 w + 3, lane l the chunks l, l + 32, ..
//           whose columns of all p_k it keeps in registers (128 of them);
//           the 16 sums of two rows are reduced over the lanes together;
//   update  thread (chunk, half) adds its 4 columns of 16 rows to 4 x 8 FP32
//           accumulators, emptied into FP64 ones every kMultiFlush tiles
//           (runs of at most 128 rows).
// 32 FMAs an element and 4 bytes: 44 us of packed FP32 FMAs against 60 us of
// HBM at 200000 x 500; a pass takes 170 us, bound by the phases' latencies.
// (Sixteen warps of four columns a lane: 220 us.  Split-TF32 matrix
// instructions: 150 us, and twice the iterations for want of precision.)
// A dot's sums are FP32 over a lane's columns and the warp's lanes, a column's
// FP32 over a run's rows; FP64 beyond, products and ut as in the one-column
// pass.
constexpr int kMultiThreads = 256;
constexpr int kMultiRows = 32;
constexpr int kMultiMaxN = 512;
constexpr int kMultiChunks = kMultiMaxN / 4;
constexpr int kMultiFlush = 8;
constexpr int kNP = kBatchMax;

__device__ __forceinline__ void mp_copy(void* dst, const void* src, int bytes) {  // 16 bytes, zeros past `bytes`
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(kMultiThreads, 1) multi_rows_kernel(MultiPass P) {
    extern __shared__ __align__(16) uint8_t msm[];
    const int n = (int)P.n, nch = (n + 3) / 4, pitch = nch * 4;
    float* tiles = reinterpret_cast<float*>(msm);                                   // 2 x 32 x pitch
    double* acc64 = reinterpret_cast<double*>(tiles + 2 * kMultiRows * pitch);      // [half][k][pitch]
    __shared__ __align__(16) float uts[kMultiRows][kNP];
    __shared__ double ssw[8][kNP];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int kk = lane & 7;  // the column whose ut this lane forms
    bool any = false;
    uint32_t on = 0;  // columns this pass serves
#pragma unroll
    for (int k = 0; k < kNP; ++k)
        if (k < P.K && (P.coef || P.st[k].done == 0)) on |= 1u << k;
    any = on != 0;
    if (!any) return;
    const double cp = kk < P.K ? (P.coef ? P.coef[0] : P.st[kk].coef[0]) : 0.0;
    const double cu = kk < P.K && P.u_in ? (P.coef ? P.coef[1] : P.st[kk].coef[1]) : 0.0;
    const bool mine = (on >> kk) & 1u;

    const int64_t per = (P.m + gridDim.x - 1) / gridDim.x;
    const int64_t r0 = (int64_t)blockIdx.x * per;
    const int64_t r1 = r0 + per < P.m ? r0 + per : P.m;
    const int rows = r1 > r0 ? (int)(r1 - r0) : 0;
    const int ntiles = (rows + kMultiRows - 1) / kMultiRows;

    float2 pv[4][2][kNP];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < kNP; ++k) {
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int col = (c * 32 + lane) * 4 + e;
                x[e] = (((on >> k) & 1u) && col < n) ? __ldg(P.p + (size_t)k * P.ps + col) : 0.0f;
            }
            pv[c][0][k] = make_float2(x[0], x[1]);
            pv[c][1][k] = make_float2(x[2], x[3]);
        }
    for (int e = t; e < 2 * kNP * pitch; e += kMultiThreads) acc64[e] = 0.0;

    auto issue = [&](int q) {
        if (q < ntiles) {
            float* dst = tiles + (q & 1) * kMultiRows * pitch;
            for (int e = t; e < kMultiRows * nch; e += kMultiThreads) {
                const int r = e / nch, c = e - r * nch;
                const int64_t row = r0 + q * kMultiRows + r;
                const int left = (n - c * 4) * 4;
                const int bytes = row < r1 ? (left < 16 ? left : 16) : 0;
                mp_copy(dst + r * pitch + c * 4, bytes ? P.A + (size_t)row * P.ld + c * 4 : P.A, bytes);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    issue(1);
    // thread's share of the update: chunk uc, rows 16 uh .. 16 uh + 15
    const int uc = t & (kMultiChunks - 1), uh = t >> 7;
    float2 acc[4][kNP / 2];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int k = 0; k < kNP / 2; ++k) acc[e][k] = make_float2(0.0f, 0.0f);
    auto flush = [&]() {
        if (uc < nch) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int k = 0; k < kNP / 2; ++k) {
                    double* d = acc64 + ((size_t)uh * kNP + 2 * k) * pitch + uc * 4 + e;
                    d[0] += (double)acc[e][k].x;
                    d[pitch] += (double)acc[e][k].y;
                    acc[e][k] = make_float2(0.0f, 0.0f);
                }
        }
    };
    double ss = 0.0;
    for (int q = 0; q < ntiles; ++q) {
        const float* tile = tiles + (q & 1) * kMultiRows * pitch;
        const int row = 4 * warp + (lane >> 3);  // the row whose ut this lane forms
        const int64_t i = r0 + q * kMultiRows + row;
        const float uin = (mine && cu != 0.0 && i < r1) ? __ldg(P.u_in + (size_t)kk * P.ui + i) : 0.0f;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float mydot = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // rows 4 w + 2 h, + 1
            float2 d[2][kNP];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int k = 0; k < kNP; ++k) d[u][k] = make_float2(0.0f, 0.0f);
            const float* base = tile + (4 * warp + 2 * h) * pitch + lane * 4;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c * 32 + lane >= nch) continue;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 a = *reinterpret_cast<const float4*>(base + u * pitch + c * 128);
                    const float2 x = make_float2(a.x, a.y), y = make_float2(a.z, a.w);
#pragma unroll
                    for (int k = 0; k < kNP; ++k) {
                        d[u][k] = __ffma2_rn(x, pv[c][0][k], d[u][k]);
                        d[u][k] = __ffma2_rn(y, pv[c][1][k], d[u][k]);
                    }
                }
            }
            // v[0..15] = (row u, column k) at 8 u + k; after the exchanges
            // lane l holds the sum over all lanes of v[l % 16]
            float v[16];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int k = 0; k < kNP; ++k) v[u * kNP + k] = d[u][k].x + d[u][k].y;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (e >= o) continue;
                    const float give = up ? v[e] : v[e + o];
                    const float keep = up ? v[e + o] : v[e];
                    v[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
            const float s = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
            if ((lane >> 4) == h) mydot = s;
        }
        const float ut = i < r1 ? (float)(cp * (double)mydot + (cu != 0.0 ? cu * (double)uin : 0.0)) : 0.0f;
        uts[row][kk] = mine ? ut : 0.0f;
        if (mine && i < r1) {
            if (P.u_out) P.u_out[(size_t)kk * P.uo + i] = ut;
            ss += (double)ut * (double)ut;
        }
        __syncthreads();
        if (uc < nch) {
#pragma unroll 4
            for (int r = 16 * uh; r < 16 * uh + 16; ++r) {
                const float4 a = *reinterpret_cast<const float4*>(tile + r * pitch + uc * 4);
                const float4 w0 = *reinterpret_cast<const float4*>(&uts[r][0]);
                const float4 w1 = *reinterpret_cast<const float4*>(&uts[r][4]);
                const float2 w[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y),
                                     make_float2(w1.z, w1.w)};
                const float x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int k = 0; k < kNP / 2; ++k) acc[e][k] = __ffma2_rn(make_float2(x[e], x[e]), w[k], acc[e][k]);
            }
        }
        if ((q + 1) % kMultiFlush == 0) flush();
        __syncthreads();  // the tile and uts may be overwritten
        issue(q + 2);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    flush();
    ss += __shfl_xor_sync(0xffffffffu, ss, 8);
    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
    if (lane < kNP) ssw[warp][lane] = ss;
    __syncthreads();
    for (int e = t; e < P.K * n; e += kMultiThreads) {
        const int k = e / n, j = e - k * n;
        if (!((on >> k) & 1u)) continue;
        P.qpart[((size_t)blockIdx.x * P.K + k) * P.qs + j] =
            (float)(acc64[(size_t)k * pitch + j] + acc64[((size_t)kNP + k) * pitch + j]);
    }
    if (P.sspart && t < P.K && ((on >> t) & 1u)) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += ssw[w][t];
        P.sspart[(size_t)t * gridDim.x + blockIdx.x] = s;
    }
}

// Partial sums of squares of the columns b_k.
__global__ void __launch_bounds__(256) batch_sumsq_kernel(const float* __restrict__ b, int64_t ldb, int64_t m,
                                                          double* __restrict__ part) {
    __shared__ double sm[32];
    const float* x = b + (size_t)blockIdx.y * ldb;
    const int64_t per = (m + gridDim.x - 1) / gridDim.x, i0 = (int64_t)blockIdx.x * per;
    const int64_t i1 = i0 + per < m ? i0 + per : m;
    double s = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) s += (double)x[i] * (double)x[i];
    s = block_sum(s, sm);
    if (threadIdx.x == 0) part[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

// ||b_k|| and ||A||_F into the states (block k: column k).
__global__ void __launch_bounds__(256) batch_norms_kernel(const double* __restrict__ part, int np,
                                                          const double* anorm_dev, LsqrDev* st) {
    __shared__ double sm[32];
    const double bn = sqrt(block_sum_array(part + (size_t)blockIdx.x * np, np, sm));
    if (threadIdx.x != 0) return;
    LsqrDev& s = st[blockIdx.x];
    s.rhsnorm = bn;
    s.bnorm = bn;
    if (anorm_dev) s.anorm_fro = *anorm_dev;
}

size_t a256(size_t b) { return (b + 255) / 256 * 256; }

// The columns' vectors inside ws->bat.
struct BatchBufs {
    float *u, *v, *wt, *p, *x, *qpart;
    double *t, *vhat, *sspart, *cpart, *scal, *bpart, *coef;
    LsqrDev* st;
    int* ticket;
    size_t bytes;
};

BatchBufs batch_layout(void* base, int64_t m, int64_t n, int64_t K, int64_t qs, int grid, int gs) {
    BatchBufs b;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* q = p ? p + off : nullptr;
        off += a256(bytes);
        return q;
    };
    const size_t k = (size_t)K;
    b.u = reinterpret_cast<float*>(take(k * m * 4));
    b.v = reinterpret_cast<float*>(take(k * n * 4));
    b.wt = reinterpret_cast<float*>(take(k * n * 4));
    b.p = reinterpret_cast<float*>(take(k * n * 4));
    b.x = reinterpret_cast<float*>(take(k * n * 4));
    b.qpart = reinterpret_cast<float*>(take((size_t)grid * k * qs * 4));
    b.t = reinterpret_cast<double*>(take(k * n * 8));
    b.vhat = reinterpret_cast<double*>(take(k * n * 8));
    b.sspart = reinterpret_cast<double*>(take(k * grid * 8));
    b.cpart = reinterpret_cast<double*>(take(k * 48 * 8));
    b.scal = reinterpret_cast<double*>(take(k * 8 * 8));
    b.bpart = reinterpret_cast<double*>(take(k * gs * 8));
    b.coef = reinterpret_cast<double*>(take(2 * 8));
    b.st = reinterpret_cast<LsqrDev*>(take(k * sizeof(LsqrDev)));
    b.ticket = reinterpret_cast<int*>(take(4));
    b.bytes = off;
    return b;
}

}  // namespace

int multi_pass_grid(int64_t m) {
    int64_t g = (m + kMultiRows - 1) / kMultiRows;
    if (g > sm_count()) g = sm_count();
    return g < 1 ? 1 : (int)g;
}

bool multi_pass_ok(const tomos_dense* A, int64_t K) {
    return A->numeric == TOMOS_FP32 && A->layout == TOMOS_ROW_MAJOR && A->rows > 0 && A->cols >= 1 &&
           A->cols <= kMultiMaxN && K >= 2 && K <= kBatchMax && A->ld % 4 == 0 &&
           reinterpret_cast<uintptr_t>(A->values) % 16 == 0;
}

tomos_status enqueue_multi_pass(const MultiPass& P, cudaStream_t st) {
    const size_t pitch = (size_t)(P.n + 3) / 4 * 4;
    const size_t smem = 2 * kMultiRows * pitch * 4 + 2 * kNP * pitch * 8;
    TOMOS_CUDA_TRY(cudaFuncSetAttribute(multi_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    multi_rows_kernel<<<multi_pass_grid(P.m), kMultiThreads, smem, st>>>(P);
    TOMOS_LAUNCH_CHECK("multi_rows_kernel");
    return TOMOS_OK;
}

}  // namespace tomos_b200

using namespace tomos_b200;

extern "C" {

int32_t tomos_lsqr_batch_supported(const tomos_dense* A, int32_t K, const tomos_workspace* ws) {
    if (!A || !ws || !multi_pass_ok(A, K) || !ws->has_precond) return 0;
    return nside_batch_ok(A->cols) ? 1 : 0;
}

tomos_status tomos_lsqr_solve_batch_dense(const tomos_dense* A, int32_t K, const float* B, int64_t ldb, float* X,
                                          int64_t ldx, tomos_workspace* ws, const tomos_lsqr_opts* o,
                                          tomos_lsqr_report* reports, void* stream) {
    std::string why;
    if (!opts_ok(o, &why)) return fail(TOMOS_ERR_INVALID, "lsqr_solve_batch: " + why);
    if (!A || !B || !X || !reports || !A->values) return fail(TOMOS_ERR_INVALID, "lsqr_solve_batch: null pointer");
    tomos_status s = workspace_check(ws, A->rows, A->cols);
    if (s) return s;
    if (A->ld < A->cols || ldb < A->rows || ldx < A->cols)
        return fail(TOMOS_ERR_INVALID, "lsqr_solve_batch: leading dimension too small");
    if (!tomos_lsqr_batch_supported(A, K, ws) || o->stop_rule != TOMOS_STOP_BACKWARD || o->comm || o->refine ||
        o->refine_csr || o->staged_plane || o->warm_start || o->implicit_duplicate || o->profile ||
        (o->iter_tier != TOMOS_TIER_AUTO && o->iter_tier != TOMOS_TIER_NATIVE) ||
        !(o->anorm_fro_dev || o->anorm_fro > 0.0))
        return fail(TOMOS_ERR_UNSUPPORTED, "lsqr_solve_batch: no batched kernel registered for these arguments");
    const int64_t m = A->rows, n = A->cols;
    const int grid = multi_pass_grid(m);
    const int64_t qs = ws->qstride;
    const BatchBufs need = batch_layout(nullptr, m, n, K, qs, grid, ws->gs_max);
    if (need.bytes > ws->bat_bytes) {
        release_memory(ws, ws->bat);
        ws->bat = nullptr;
        ws->bat_bytes = 0;
        if (pool_malloc(&ws->bat, need.bytes) != cudaSuccess) {
            cudaGetLastError();
            return fail(TOMOS_ERR_ALLOC, "lsqr_solve_batch: workspace allocation failed");
        }
        ws->bat_bytes = need.bytes;
    }
    const BatchBufs b = batch_layout(ws->bat, m, n, K, qs, grid, ws->gs_max);
    PassPlan pl_init = plan_dense_pass(ws, A, Elem::F32, true, o->tol >= kRunsTolMin);
    if (pass_needs_scratch(pl_init)) {
        s = ensure_scratch(ws, dense_pass_scratch(A));
        if (s) return s;
    }
    cudaStream_t us = as_stream(stream), st = ws->stream;
    TOMOS_CUDA_TRY(cudaEventRecord(ws->ev_fence, us));
    TOMOS_CUDA_TRY(cudaStreamWaitEvent(st, ws->ev_fence, 0));
    TOMOS_CUDA_TRY(cudaEventRecord(ws->ev_start, st));
    const int64_t launches0 = ws->launches;
    s = refresh_precond(ws, st);
    if (s) return s;
    TOMOS_CUDA_TRY(cudaMemsetAsync(b.x, 0, sizeof(float) * (size_t)K * n, st));
    TOMOS_CUDA_TRY(cudaMemsetAsync(b.ticket, 0, sizeof(int), st));
    const double* dsc = nullptr;
    if (o->col_scale) {
        TOMOS_CUDA_TRY(cudaMemcpyAsync(ws->dscale, o->col_scale, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        dsc = ws->dscale;
    }
    const int max_iters = o->max_iters > 0 ? o->max_iters : 0;
    const int restarts = o->restarts > 0 ? o->restarts : 1;
    std::vector<LsqrDev> H((size_t)K);
    std::memset(H.data(), 0, sizeof(LsqrDev) * K);
    for (LsqrDev& h : H) {
        h.anorm_fro = o->anorm_fro;
        h.tol = o->tol;
        h.max_relres = o->max_relres;
        h.inner_rtol = o->inner_rtol;
        h.inner_tol = o->tol * (o->inner_eta_factor > 0.0 ? o->inner_eta_factor : 1.0);
        h.max_iters = max_iters;
        h.stop_rule = o->stop_rule;
        h.done = 1;
    }
    TOMOS_CUDA_TRY(cudaMemcpyAsync(b.st, H.data(), sizeof(LsqrDev) * K, cudaMemcpyHostToDevice, st));
    const double coef[2] = {-1.0, 1.0};
    TOMOS_CUDA_TRY(cudaMemcpyAsync(b.coef, coef, sizeof(coef), cudaMemcpyHostToDevice, st));
    for (int k = 0; k < K; ++k)  // ws->scal[7]: whether R^{-1} has a lower triangle (refresh_precond)
        TOMOS_CUDA_TRY(cudaMemcpyAsync(b.scal + 8 * k + 7, ws->scal + 7, sizeof(double), cudaMemcpyDeviceToDevice, st));
    batch_sumsq_kernel<<<dim3((unsigned)ws->gs_max, (unsigned)K), 256, 0, st>>>(B, ldb, m, b.bpart);
    TOMOS_LAUNCH_CHECK("batch_sumsq_kernel");
    batch_norms_kernel<<<(unsigned)K, 256, 0, st>>>(b.bpart, ws->gs_max, o->anorm_fro_dev, b.st);
    TOMOS_LAUNCH_CHECK("batch_norms_kernel");
    ws->launches += 2;

    MultiPass mp;
    mp.A = static_cast<const float*>(A->values);
    mp.m = m;
    mp.n = n;
    mp.ld = A->ld;
    mp.K = K;
    mp.p = b.p;
    mp.ps = n;
    mp.u_in = b.u;
    mp.ui = m;
    mp.u_out = b.u;
    mp.uo = m;
    mp.coef = nullptr;
    mp.st = b.st;
    mp.qpart = b.qpart;
    mp.qs = qs;
    mp.sspart = b.sspart;
    PassPlan pl_multi;
    pl_multi.gq = grid;
    pl_multi.gs = grid;
    pl_multi.qstride = (int64_t)K * qs;
    // column k's n-side; single: its partials are those of a one-column pass
    auto nside = [&](int k, const PassPlan& pl, bool init, bool single) {
        NSide S = make_nside(ws, pl, b.x + (size_t)k * n, init, init ? nullptr : &b.st[k].done, dsc);
        S.t = b.t + (size_t)k * n;
        S.vhat = b.vhat + (size_t)k * n;
        S.v = b.v + (size_t)k * n;
        S.wt = b.wt + (size_t)k * n;
        S.p = b.p + (size_t)k * n;
        S.scal = b.scal + 8 * (size_t)k;
        S.cpart = b.cpart + 48 * (size_t)k;
        S.st = b.st + k;
        if (!single) {
            S.qpart = b.qpart + (size_t)k * qs;
            S.sspart = b.sspart + (size_t)k * grid;
        }
        return S;
    };
    NSide S[kBatchMax];

    // one launch runs a cycle's iterations: a while loop over the shared pass
    // and the columns' n-side, ended by the last column's stopping rule
    const std::vector<uint64_t> key = {reinterpret_cast<uint64_t>(A->values), (uint64_t)A->ld, (uint64_t)K,
                                       reinterpret_cast<uint64_t>(ws->bat), reinterpret_cast<uint64_t>(dsc),
                                       reinterpret_cast<uint64_t>(ws->Rcm)};
    if (!ws->bgraph || ws->bgraph_key != key) {
        if (ws->bgraph) cudaGraphExecDestroy(ws->bgraph);
        ws->bgraph = nullptr;
        const int64_t before = ws->launches;
        cudaGraph_t g = nullptr;
        cudaGraphConditionalHandle h = 0;
        cudaGraphNodeParams cp = {};
        cudaGraphNode_t node = nullptr;
        bool ok = cudaGraphCreate(&g, 0) == cudaSuccess &&
                  cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
        if (ok) {
            cp.type = cudaGraphNodeTypeConditional;
            cp.conditional.handle = h;
            cp.conditional.type = cudaGraphCondTypeWhile;
            cp.conditional.size = 1;
            ok = cudaGraphAddNode(&node, g, nullptr, 0, &cp) == cudaSuccess;
        }
        if (ok)
            ok = cudaStreamBeginCaptureToGraph(st, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        if (ok) {
            tomos_status cs = enqueue_multi_pass(mp, st);
            for (int k = 0; k < K; ++k) {
                S[k] = nside(k, pl_multi, false, false);
                S[k].cond = h;
                S[k].use_cond = 1;
                S[k].ticket = b.ticket;
                S[k].group = K;
                S[k].group_st = b.st;
            }
            if (!cs) cs = enqueue_nside_batch(ws, S, K, st);
            cudaGraph_t body = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(st, &body);
            if (cs) {
                cudaGraphDestroy(g);
                return cs;
            }
            ok = ce == cudaSuccess;
        }
        if (ok) ok = cudaGraphInstantiate(&ws->bgraph, g, 0) == cudaSuccess;
        if (g) cudaGraphDestroy(g);
        ws->launches = before;
        if (!ok) {
            cudaGetLastError();
            ws->bgraph = nullptr;
            return fail(TOMOS_ERR_UNSUPPORTED, "lsqr_solve_batch: conditional graphs unavailable");
        }
        ws->bgraph_key = key;
        ws->bgraph_kernels = 2;
    }

    auto sync_states = [&]() -> tomos_status {
        TOMOS_CUDA_TRY(cudaMemcpyAsync(H.data(), b.st, sizeof(LsqrDev) * K, cudaMemcpyDeviceToHost, st));
        TOMOS_CUDA_TRY(cudaMemcpyAsync(ws->st_host, ws->st, sizeof(LsqrDev), cudaMemcpyDeviceToHost, st));
        TOMOS_CUDA_TRY(cudaStreamSynchronize(st));
        if (ws->st_host->pipe_err)
            return fail(TOMOS_ERR_CUDA, "A pass: a bounded pipeline wait expired (code " +
                                            std::to_string(ws->st_host->pipe_err) + ")");
        return TOMOS_OK;
    };
    TOMOS_CUDA_TRY(cudaMemsetAsync(ws->st, 0, sizeof(LsqrDev), st));  // the one-column passes' error word
    // column k's accurate pass from its x (the residual that certifies it)
    auto accurate = [&](int k) -> tomos_status {
        struct SwapU {  // the one-column pass writes ws->u
            tomos_workspace* w;
            float* old;
            ~SwapU() { w->u = old; }
        } swap{ws, ws->u};
        ws->u = b.u + (size_t)k * m;
        tomos_status e = enqueue_dense_pass(ws, A, pl_init, b.x + (size_t)k * n, B + (size_t)k * ldb, b.coef, nullptr, st);
        if (e) return e;
        return enqueue_nside(ws, nside(k, pl_init, true, true), st);
    };
    std::memset(reports, 0, sizeof(tomos_lsqr_report) * K);
    std::vector<char> finished((size_t)K, 0);
    auto check = [&](int k) {
        tomos_lsqr_report& R = reports[k];
        const LsqrDev& h = H[(size_t)k];
        if (h.rhsnorm == 0.0) {
            R.converged = 1;
            return true;
        }
        R.rnorm = h.beta;
        R.arnorm = h.arnorm;
        R.xnorm = h.xnorm;
        R.backward_error = eta_of(h);
        if (R.backward_error <= o->tol || h.beta == 0.0) R.converged = 1;
        return R.converged != 0;
    };
    for (int rs = 0; rs < restarts; ++rs) {
        if (rs == 0) {  // from x = 0 the pass only forms A^T b
            MultiPass m0 = mp;
            m0.p = b.x;
            m0.u_in = B;
            m0.ui = ldb;
            m0.coef = b.coef;
            s = enqueue_multi_pass(m0, st);
            if (s) return s;
            for (int k = 0; k < K; ++k) S[k] = nside(k, pl_multi, true, false);
            s = enqueue_nside_batch(ws, S, K, st);
            if (s) return s;
            ws->launches += 1;
        } else {
            for (int k = 0; k < K; ++k)
                if (!finished[(size_t)k]) {
                    s = accurate(k);
                    if (s) return s;
                    reports[k].accurate_passes += 1;
                }
        }
        s = sync_states();
        if (s) return s;
        int going = 0;
        for (int k = 0; k < K; ++k) {
            if (finished[(size_t)k]) continue;
            reports[k].restarts_used = rs + 1;
            if (rs == 0) reports[k].half_passes += 1;
            if (check(k)) finished[(size_t)k] = 1;
            if (finished[(size_t)k] || H[(size_t)k].breakdown || max_iters == 0)
                TOMOS_CUDA_TRY(cudaMemsetAsync(&b.st[k].done, 1, sizeof(int), st));  // nonzero: idle this cycle
            else
                ++going;
        }
        bool all = true;
        for (char f : finished) all = all && f;
        if (all) break;
        if (!going) continue;
        const std::vector<LsqrDev> before = H;
        TOMOS_CUDA_TRY(cudaGraphLaunch(ws->bgraph, st));
        s = sync_states();
        if (s) return s;
        int most = 0;
        for (int k = 0; k < K; ++k) {
            const int it = H[(size_t)k].iter - before[(size_t)k].iter;
            if (it > 0) reports[k].half_passes += it;
            if (it > most) most = it;
        }
        ws->launches += (int64_t)most * ws->bgraph_kernels;
    }
    bool rest = false;
    for (int k = 0; k < K; ++k)
        if (!finished[(size_t)k]) {
            s = accurate(k);
            if (s) return s;
            reports[k].accurate_passes += 1;
            rest = true;
        }
    if (rest) {
        s = sync_states();
        if (s) return s;
        for (int k = 0; k < K; ++k)
            if (!finished[(size_t)k]) check(k);
    }
    for (int k = 0; k < K; ++k)
        TOMOS_CUDA_TRY(cudaMemcpyAsync(X + (size_t)k * ldx, b.x + (size_t)k * n, sizeof(float) * n,
                                       cudaMemcpyDeviceToDevice, st));
    TOMOS_CUDA_TRY(cudaEventRecord(ws->ev_stop, st));
    TOMOS_CUDA_TRY(cudaEventSynchronize(ws->ev_stop));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ws->ev_start, ws->ev_stop);
    TOMOS_CUDA_TRY(cudaEventRecord(ws->ev_fence, st));
    TOMOS_CUDA_TRY(cudaStreamWaitEvent(us, ws->ev_fence, 0));
    for (int k = 0; k < K; ++k) {
        tomos_lsqr_report& R = reports[k];
        const LsqrDev& h = H[(size_t)k];
        R.iterations = h.iter;
        R.relres = h.relres;
        R.anorm_fro = h.anorm_fro;
        R.bnorm = h.bnorm;
        R.elapsed_ms = ms;
        R.kernel_launches = (int32_t)(ws->launches - launches0);
    }
    return TOMOS_OK;
}

}  // extern "C"
