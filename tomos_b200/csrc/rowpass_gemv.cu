// rowpass_gemv.cu -- tomos_gemv through the row pass (rowpass.cuh).
//
// A strided product y = alpha op(A) x + beta y is, over the lines of A
// (rows of a row-major A, columns of a column-major one), either a dot per
// line or a sum of scaled lines (gemv.cu).  When the lines are 16-byte
// aligned and short enough for the consumer warps, both shapes stream every
// line through shared memory once with bulk asynchronous copies, as the
// LSQR pass does, and decode the storage in registers:
//   dot per line      kRowDot:  y_o = alpha (A_o . x) + beta y_o, one
//                     warp (or G warps) per line, written in place;
//   sum of lines      kRowAxpy: per-CTA partials of sum_o x_o A_o, then
//                     sum_parts_kernel (gemv.cu) sums the partials of
//                     every column in a fixed order (deterministic, no
//                     atomics; the reference adds with atomicAdd,
//                     mv_cuda_kernels.cu:529) into y = alpha sum + beta y.
// Narrow lines, and lines that do not start on 16-byte boundaries, take the
// direct pass (rowpass_direct.cuh) instead, where it is the better one.
// FP32 and HALF-tier products accumulate in FP32.  The exact tiers form
// FP32 products over short runs (a lane's part of a line, or 8 lines of a
// column) and sum the runs in FP64.  Other shapes take the generic
// kernels of gemv.cu.
#include <mutex>
#include <string>

#include "common.cuh"
#include "gemv.cuh"
#include "rowpass_direct.cuh"
#include "rowpass_launch.cuh"

namespace tomos_b200 {

namespace {

// The word a bounded pipeline wait of these launches records its expiry
// in (one per device; nothing reads it back: an expired wait leaves the
// product's y undefined, which the bounded waits make the only effect of
// a stalled copy).
__device__ int g_rowpass_gemv_err;
constexpr int kMaxDevices = 64;

int* err_word() {
    static std::mutex mu;
    static int* addr[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_rowpass_gemv_err) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        addr[dev] = static_cast<int*>(p);
    }
    return addr[dev];
}

template <int MODE>
tomos_status launch_mode(Elem e, bool acc64, const FusedParams& P, int* err, int nch, int g, int grid,
                         cudaStream_t st, double* qpart64) {
    switch (e) {
        case Elem::F32: return launch_fused_e<Elem::F32, false, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::H16: return launch_fused_e<Elem::H16, false, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::F16: return launch_fused_e<Elem::F16, false, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::B16: return launch_fused_e<Elem::B16, false, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::A16: return launch_fused_e<Elem::A16, true, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::AB16: return launch_fused_e<Elem::AB16, true, MODE>(P, err, nch, g, grid, st, qpart64);
        case Elem::AB16R: return launch_fused_e<Elem::AB16R, true, MODE>(P, err, nch, g, grid, st, qpart64);
        default: return fail(TOMOS_ERR_UNSUPPORTED, "gemv row pass: element type");
    }
}

}  // namespace

size_t rowpass_gemv_scratch_bytes(int64_t outer, int64_t inner) {
    const int64_t qs = (inner + 31) / 32 * 32;
    int64_t rows = sm_count();
    if (inner <= kDirectMaxCols && direct_grid(outer) > rows) rows = direct_grid(outer);
    return (size_t)rows * (size_t)qs * sizeof(double);
}

// Whether the direct pass forms a product of lines it covers.  Sums of very
// few lines, and the dots of few, are shorter in the generic kernels (gemv.cu;
// a warp a line for dots), which start faster (times warm in L2):
//   sums   8 lines of 1000 FP32 3.5 us (direct 5.3), 64 lines 7.0 us (5.1);
//   dots   3000 lines of 64 aligned FP32 2.1 us (3.6), 10000 3.5 us (3.8);
//          unaligned: 3000 lines of 65 FP32 2.2 us (4.2), 30000 6.4 us (5.5);
//          777 at 30000 19.2 us (18.7); exact FP32_16 of 500 at 30000 31 us
//          (33), at 100000 152 us (105);
// and so are the dots of 16-bit lines whose chunks leave the 32 lanes' slots
// half empty: 100000 lines of 257 exact FP32_16 77 us (101), FP16 21 us (23).
static bool direct_better(const GemvLaunch& L, Elem e, const DirectShape& ds) {
    if (!L.dot) return L.outer >= 24;
    if (direct_aligned(e, L.ld, L.hi, L.lo) || (e == Elem::H16 && L.inner > 256)) return L.outer >= 10000;
    if (L.outer < (ds.c > 1 || (elem_is_exact(e) && ds.lpr > 8) ? 40000 : 24000)) return false;
    const int64_t nch = (L.inner + 14) / 8;
    return e == Elem::F32 || e == Elem::H16 || ds.lpr < 32 || 10 * nch >= 7 * 32 * ds.c;
}

// The product through the direct pass (*used false: scratch too small).
static tomos_status direct_gemv(const GemvLaunch& L, Elem e, const DirectShape& ds, cudaStream_t st, bool* used) {
    const bool acc64 = elem_is_exact(e);
    // sums of narrow lines: 64 lines a CTA at least, which leaves fewer partials
    // (300 lines of 20 FP32: 4.8 us, with 16 lines a CTA 5.9 us)
    int grid = direct_grid(L.outer);
    if (!L.dot && ds.lpr < 32 && grid > (L.outer + 63) / 64) grid = (int)((L.outer + 63) / 64);
    const int64_t qs = (L.inner + 31) / 32 * 32;
    if (!L.dot && (!L.scratch || L.scratch_bytes < (size_t)grid * qs * (acc64 ? 8 : 4))) return TOMOS_OK;
    *used = true;
    DirectParams T;
    FusedParams& P = T.f;
    P.hi = L.hi;
    P.lo = L.lo;
    P.m = L.outer;
    P.n = L.inner;
    P.ld = L.ld;
    P.coef = nullptr;
    P.sspart = nullptr;
    P.skip = nullptr;
    P.qstride = qs;
    T.dot = L.dot ? 1 : 0;
    T.axpy = L.dot ? 0 : 1;
    T.write_u = T.dot;
    T.aligned = direct_aligned(e, L.ld, L.hi, L.lo) ? 1 : 0;
    P.p = L.dot ? L.x : nullptr;
    P.u_in = L.dot ? L.y : L.x;
    P.u_out = L.dot ? L.y : nullptr;
    P.cp = L.dot ? L.alpha : 0.0;
    P.cu = L.dot ? L.beta : 1.0;
    P.qpart = static_cast<float*>(L.scratch);
    T.qpart64 = static_cast<double*>(L.scratch);
    tomos_status s = launch_direct(e, acc64, T, ds, grid, st);
    if (s || L.dot) return s;
    return acc64 ? launch_sum_parts(T.qpart64, grid, qs, L.inner, L.alpha, L.beta, nullptr, nullptr, L.y, st)
                 : launch_sum_parts(P.qpart, grid, qs, L.inner, L.alpha, L.beta, nullptr, nullptr, L.y, st);
}

tomos_status rowpass_gemv(const GemvLaunch& L, Elem e, cudaStream_t st, bool* used) {
    *used = false;
    const bool acc64 = elem_is_exact(e);
    if (e == Elem::F64 || L.coef || L.skip) return TOMOS_OK;
    const DirectShape ds = direct_shape(e, L.inner, L.ld, L.hi, L.lo);
    if (ds.lpr > 0) return direct_better(L, e, ds) ? direct_gemv(L, e, ds, st, used) : TOMOS_OK;
    int nch = 0, g = 1;
    if (!plan_row_lines(e, acc64, L.dot ? kRowDot : kRowAxpy, L.inner, L.ld, L.hi, L.lo, &nch, &g)) return TOMOS_OK;
    const int grid = row_pass_grid(L.outer);
    const int64_t qs = (L.inner + 31) / 32 * 32;
    if (!L.dot && (!L.scratch || L.scratch_bytes < (size_t)grid * qs * (acc64 ? 8 : 4))) return TOMOS_OK;
    int* err = err_word();
    if (!err) return TOMOS_OK;
    *used = true;
    FusedParams P;
    P.hi = L.hi;
    P.lo = L.lo;
    P.m = L.outer;
    P.n = L.inner;
    P.ld = L.ld;
    P.coef = nullptr;
    P.sspart = nullptr;
    P.skip = nullptr;
    P.qstride = qs;
    if (L.dot) {
        // y_o = alpha (A_o . x) + beta y_o, in place (y is not read when beta == 0)
        P.p = L.x;
        P.u_in = L.y;
        P.u_out = L.y;
        P.qpart = nullptr;
        P.cp = L.alpha;
        P.cu = L.beta;
        return launch_mode<kRowDot>(e, acc64, P, err, nch, g, grid, st, nullptr);
    }
    // partials of sum_o x_o A_o, then y = alpha sum + beta y
    P.p = nullptr;
    P.u_in = L.x;
    P.u_out = nullptr;
    P.cp = 0.0;
    P.cu = 1.0;
    P.qpart = acc64 ? nullptr : static_cast<float*>(L.scratch);
    double* q64 = acc64 ? static_cast<double*>(L.scratch) : nullptr;
    tomos_status s = launch_mode<kRowAxpy>(e, acc64, P, err, nch, g, grid, st, q64);
    if (s) return s;
    return acc64 ? launch_sum_parts(q64, grid, qs, L.inner, L.alpha, L.beta, nullptr, nullptr, L.y, st)
                 : launch_sum_parts(P.qpart, grid, qs, L.inner, L.alpha, L.beta, nullptr, nullptr, L.y, st);
}

}  // namespace tomos_b200
