// gemv.cu -- strided GEMV y = alpha * op(A) x + beta * y for every storage
// type, layout and leading dimension (tomos_gemv), and the same kernels
// with device-resident alpha/beta for the solver's unfused path.
//
// A strided matrix is `outer` lines of `inner` contiguous elements.  An
// op(A) product is then one of two shapes:
//   line dots  (row-major NO_TRANSPOSE, col-major TRANSPOSE):
//       y[o] = sum_i A[o, i] x[i]      -- a warp per line, or a CTA per
//                                         segment of a few long lines
//   line sums  (row-major TRANSPOSE, col-major NO_TRANSPOSE):
//       y[i] = sum_o A[o, i] x[o]      -- threads own i; blocks own a
//                                         chunk of lines and write partials
//                                         that a second kernel reduces in
//                                         a fixed order (deterministic, no
//                                         atomics; the reference uses
//                                         atomicAdd, mv_cuda_kernels.cu:529)
// HALF-tier and FP32 products accumulate in FP32, ACCURATE-tier in FP64.
// The row passes (rowpass.cuh, rowpass_direct.cuh) take row-major LSQR
// iterations and the products whose lines fit them; these kernels serve the
// rest.
#include <mutex>
#include <string>

#include "common.cuh"
#include "fused.cuh"
#include "gemv.cuh"

namespace tomos_b200 {

template <bool ACC64>
struct AccT {
    using T = float;
};
template <>
struct AccT<true> {
    using T = double;
};

__device__ __forceinline__ void resolve_coef(const double* coef, double& alpha, double& beta) {
    if (coef) {
        alpha = coef[0];
        beta = coef[1];
    }
}

// V consecutive elements at each of the flat indices idx + u step as floats:
// V = ChunkElems (one 16-byte load a plane, aligned) or 1.
template <Elem E, int V, int U>
__device__ __forceinline__ void load_chunks(const void* hi, const void* lo, size_t idx, size_t step, float (&f)[U][V]) {
    if constexpr (V == 1) {
        float v[U];
        load_elems<E, U>(hi, lo, idx, step, v);
#pragma unroll
        for (int u = 0; u < U; ++u) f[u][0] = v[u];
    } else {
        FusedParams P;
        P.hi = hi;
        P.lo = lo;
        uint4 h[U], l[U];
#pragma unroll
        for (int u = 0; u < U; ++u) ChunkDecoder<E>::load(P, idx + u * step, h[u], l[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) ChunkDecoder<E>::decode(h[u], l[u], f[u]);
    }
}

// Line dots, a warp per line: y[o] = alpha A_o . x + beta y[o].
template <Elem E, bool ACC64>
__global__ void __launch_bounds__(256) line_dot_kernel(const void* __restrict__ hi,
                                                       const void* __restrict__ lo,
                                                       int64_t outer, int64_t inner, int64_t ld,
                                                       const float* __restrict__ x, double alpha,
                                                       double beta, const double* coef,
                                                       const int* skip, float* __restrict__ y) {
    if (skip && *skip) return;
    using Acc = typename AccT<ACC64>::T;
    resolve_coef(coef, alpha, beta);
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t o = warp; o < outer; o += nwarps) {
        const size_t base = (size_t)o * (size_t)ld;
        Acc a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        int64_t i = lane;
        for (; i + 96 < inner; i += 128) {
            if constexpr (E == Elem::H16) {
                float v[4];
                load_elems<E, 4>(hi, lo, base + i, 32, v);
                a0 += (Acc)v[0] * (Acc)__ldg(x + i);
                a1 += (Acc)v[1] * (Acc)__ldg(x + i + 32);
                a2 += (Acc)v[2] * (Acc)__ldg(x + i + 64);
                a3 += (Acc)v[3] * (Acc)__ldg(x + i + 96);
            } else {
                a0 += (Acc)load_elem<E>(hi, lo, base + i) * (Acc)__ldg(x + i);
                a1 += (Acc)load_elem<E>(hi, lo, base + i + 32) * (Acc)__ldg(x + i + 32);
                a2 += (Acc)load_elem<E>(hi, lo, base + i + 64) * (Acc)__ldg(x + i + 64);
                a3 += (Acc)load_elem<E>(hi, lo, base + i + 96) * (Acc)__ldg(x + i + 96);
            }
        }
        for (; i < inner; i += 32) a0 += (Acc)load_elem<E>(hi, lo, base + i) * (Acc)__ldg(x + i);
        Acc acc = warp_sum((a0 + a1) + (a2 + a3));
        if (lane == 0) {
            double r = alpha * (double)acc;
            if (beta != 0.0) r += beta * (double)y[o];
            y[o] = (float)r;
        }
    }
}

// Line dots of few, long lines: a CTA per segment of a line, whose partial
// (FP64 over the CTA's lanes) sum_parts_kernel adds in segment order.  A
// warp a line left most SMs idle: 790 us for 300 lines of 100000 fp16 words,
// 33 us in segments.
template <Elem E, bool ACC64, int V>
__global__ void __launch_bounds__(256) line_dot_seg_kernel(const void* __restrict__ hi,
                                                           const void* __restrict__ lo, int64_t inner,
                                                           int64_t ld, const float* __restrict__ x,
                                                           int64_t seg, int64_t outer, const int* skip,
                                                           double* __restrict__ partial) {
    if (skip && *skip) return;
    using Acc = typename AccT<ACC64>::T;
    __shared__ double sm[8];
    const int64_t o = blockIdx.x, i0 = (int64_t)blockIdx.y * seg;  // seg: a multiple of 256 V
    const int64_t i1 = i0 + seg < inner ? i0 + seg : inner;
    const size_t base = (size_t)o * (size_t)ld;
    Acc a[4] = {0, 0, 0, 0};
    int64_t i = i0 + (int64_t)threadIdx.x * V;
    const bool xvec = reinterpret_cast<uintptr_t>(x) % 16 == 0;  // k is a multiple of V
    auto step = [&](int64_t k, Acc& acc, const float* f) {
        float xv[V];
        if (V % 4 == 0 && xvec) {
#pragma unroll
            for (int e = 0; e + 3 < V; e += 4) {
                const float4 t = __ldg(reinterpret_cast<const float4*>(x + k + e));
                xv[e] = t.x;
                xv[e + 1] = t.y;
                xv[e + 2] = t.z;
                xv[e + 3] = t.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < V; ++e) xv[e] = __ldg(x + k + e);
        }
#pragma unroll
        for (int e = 0; e < V; ++e) acc += (Acc)f[e] * (Acc)xv[e];
    };
    for (; i + 3 * 256 * V + V <= i1; i += 4 * 256 * V) {
        float f[4][V];
        load_chunks<E, V, 4>(hi, lo, base + i, 256 * V, f);
#pragma unroll
        for (int u = 0; u < 4; ++u) step(i + u * 256 * V, a[u], f[u]);
    }
    for (; i < i1; i += 256 * V) {
        if (i + V <= i1) {
            float f[1][V];
            load_chunks<E, V, 1>(hi, lo, base + i, 0, f);
            step(i, a[0], f[0]);
        } else {
            for (int64_t k = i; k < i1; ++k) a[0] += (Acc)load_elem<E>(hi, lo, base + k) * (Acc)__ldg(x + k);
        }
    }
    const double d = warp_sum((double)((a[0] + a[1]) + (a[2] + a[3])));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += sm[w];
        partial[(size_t)blockIdx.y * outer + o] = t;
    }
}

// Line sums: a thread owns V consecutive elements of the lines of its
// chunk, eight lines' loads in flight.
template <Elem E, bool ACC64, int V>
__global__ void __launch_bounds__(256) line_sum_partial_kernel(
    const void* __restrict__ hi, const void* __restrict__ lo, int64_t outer, int64_t inner,
    int64_t ld, const float* __restrict__ x, int64_t lines_per_chunk, const int* skip,
    typename AccT<ACC64>::T* __restrict__ partial) {
    if (skip && *skip) return;
    using Acc = typename AccT<ACC64>::T;
    constexpr int U = V == 1 ? 8 : 4;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * V;
    const int64_t c = blockIdx.y;
    if (i >= inner) return;
    const int64_t o0 = c * lines_per_chunk;
    int64_t o1 = o0 + lines_per_chunk;
    if (o1 > outer) o1 = outer;
    if (V > 1 && i + V > inner) {  // the last, partly filled chunk
        for (int64_t k = i; k < inner; ++k) {
            Acc a = 0;
            for (int64_t o = o0; o < o1; ++o) a += (Acc)load_elem<E>(hi, lo, (size_t)o * ld + k) * (Acc)__ldg(x + o);
            partial[(size_t)c * inner + k] = a;
        }
        return;
    }
    Acc a[2][V];
#pragma unroll
    for (int e = 0; e < V; ++e) a[0][e] = a[1][e] = 0;
    int64_t o = o0;
    for (; o + U <= o1; o += U) {
        float f[U][V];
        load_chunks<E, V, U>(hi, lo, (size_t)o * ld + i, (size_t)ld, f);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const Acc xv = (Acc)__ldg(x + o + u);
#pragma unroll
            for (int e = 0; e < V; ++e) a[u & 1][e] += (Acc)f[u][e] * xv;
        }
    }
    for (; o < o1; ++o) {
        float f[1][V];
        load_chunks<E, V, 1>(hi, lo, (size_t)o * ld + i, 0, f);
        const Acc xv = (Acc)__ldg(x + o);
#pragma unroll
        for (int e = 0; e < V; ++e) a[0][e] += (Acc)f[0][e] * xv;
    }
#pragma unroll
    for (int e = 0; e < V; ++e) partial[(size_t)c * inner + i + e] = a[0][e] + a[1][e];
}

// A CTA owns 32 columns; its warps (up to 32) split the partials, each
// thread with eight loads in flight, and sum what they hold in warp order.
// Bound by the latency of one thread's share: a thread a column took 136 us
// for 1173 partials of 777 columns.
template <typename Acc>
__global__ void __launch_bounds__(1024) sum_parts_kernel(const Acc* __restrict__ part, int64_t nparts,
                                                         int64_t stride, int64_t n, double alpha, double beta,
                                                         const double* coef, const int* skip,
                                                         float* __restrict__ y) {
    if (skip && *skip) return;
    resolve_coef(coef, alpha, beta);
    __shared__ double sm[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * 32 + lane;
    double s = 0.0;
    if (j < n) {
        int64_t c = w;
        for (; c + 7 * nw < nparts; c += 8 * nw) {
            Acc v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = part[(size_t)(c + u * nw) * stride + j];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += (double)v[u];
        }
        for (; c < nparts; c += nw) s += (double)part[(size_t)c * stride + j];
    }
    sm[w][lane] = s;
    __syncthreads();
    if (w != 0 || j >= n) return;
    double t = 0.0;
    for (int k = 0; k < nw; ++k) t += sm[k][lane];
    double r = alpha * t;
    if (beta != 0.0) r += beta * (double)y[j];
    y[j] = (float)r;
}

// Few partials: a thread a column.
template <typename Acc>
__global__ void __launch_bounds__(256) sum_few_parts_kernel(const Acc* __restrict__ part, int64_t nparts,
                                                            int64_t stride, int64_t n, double alpha, double beta,
                                                            const double* coef, const int* skip,
                                                            float* __restrict__ y) {
    if (skip && *skip) return;
    resolve_coef(coef, alpha, beta);
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double r = alpha * sum_few(part + j, nparts, stride);
    if (beta != 0.0) r += beta * (double)y[j];
    y[j] = (float)r;
}

template <typename Acc>
static tomos_status sum_parts(const Acc* part, int64_t nparts, int64_t stride, int64_t n, double alpha,
                              double beta, const double* coef, const int* skip, float* y, cudaStream_t st) {
    if (few_parts(nparts, n)) {
        sum_few_parts_kernel<Acc><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(part, nparts, stride, n, alpha, beta,
                                                                               coef, skip, y);
        TOMOS_LAUNCH_CHECK("sum_few_parts_kernel");
        return TOMOS_OK;
    }
    int64_t warps = (nparts + 7) / 8;
    if (warps > 32) warps = 32;
    sum_parts_kernel<Acc><<<(unsigned)((n + 31) / 32), (unsigned)warps * 32, 0, st>>>(part, nparts, stride, n, alpha,
                                                                                     beta, coef, skip, y);
    TOMOS_LAUNCH_CHECK("sum_parts_kernel");
    return TOMOS_OK;
}

tomos_status launch_sum_parts(const float* part, int64_t nparts, int64_t stride, int64_t n, double alpha,
                              double beta, const double* coef, const int* skip, float* y, cudaStream_t st) {
    return sum_parts(part, nparts, stride, n, alpha, beta, coef, skip, y, st);
}
tomos_status launch_sum_parts(const double* part, int64_t nparts, int64_t stride, int64_t n, double alpha,
                              double beta, const double* coef, const int* skip, float* y, cudaStream_t st) {
    return sum_parts(part, nparts, stride, n, alpha, beta, coef, skip, y, st);
}

// Chunks of the line sums' scratch: of 128 lines, at most 1184.
int64_t line_sum_chunks(int64_t outer) {
    int64_t c = (outer + 127) / 128;
    if (c > 1184) c = 1184;
    return c < 1 ? 1 : c;
}

// Segments of a line's dot: 1 while a warp per line fills the GPU (eight
// warps an SM), else enough CTAs for four an SM, of at least 8192 elements.
static int64_t line_dot_segments(int64_t outer, int64_t inner) {
    if (outer >= (int64_t)sm_count() * 8) return 1;
    int64_t g = ((int64_t)sm_count() * 4 + outer - 1) / (outer > 0 ? outer : 1);
    if (g > (inner + 8191) / 8192) g = (inner + 8191) / 8192;
    return g < 1 ? 1 : g;
}

template <Elem E, bool ACC64, int V>
static tomos_status run_gemv_v(const GemvLaunch& L, cudaStream_t st) {
    using Acc = typename AccT<ACC64>::T;
    if (L.dot) {
        const int64_t segs = line_dot_segments(L.outer, L.inner);
        // (a scratch that cannot hold doubles: a warp a line, which needs none)
        if (segs > 1 && L.scratch && reinterpret_cast<uintptr_t>(L.scratch) % sizeof(double) == 0 &&
            L.scratch_bytes >= (size_t)segs * L.outer * sizeof(double)) {
            const int64_t unit = 256 * V;
            const int64_t seg = ((L.inner + segs - 1) / segs + unit - 1) / unit * unit;
            const int64_t ns = (L.inner + seg - 1) / seg;
            double* partial = static_cast<double*>(L.scratch);
            line_dot_seg_kernel<E, ACC64, V><<<dim3((unsigned)L.outer, (unsigned)ns), 256, 0, st>>>(
                L.hi, L.lo, L.inner, L.ld, L.x, seg, L.outer, L.skip, partial);
            TOMOS_LAUNCH_CHECK("line_dot_seg_kernel");
            return sum_parts(partial, ns, L.outer, L.outer, L.alpha, L.beta, L.coef, L.skip, L.y, st);
        }
        int64_t blocks = (L.outer + 7) / 8;
        int64_t cap = (int64_t)sm_count() * 8;
        if (blocks > cap) blocks = cap;
        if (blocks < 1) blocks = 1;
        line_dot_kernel<E, ACC64><<<(unsigned)blocks, 256, 0, st>>>(
            L.hi, L.lo, L.outer, L.inner, L.ld, L.x, L.alpha, L.beta, L.coef, L.skip, L.y);
        TOMOS_LAUNCH_CHECK("line_dot_kernel");
        return TOMOS_OK;
    }
    const int64_t xb = (L.inner + 256 * V - 1) / (256 * V);
    int64_t nchunks = line_sum_chunks(L.outer);
    size_t need = (size_t)nchunks * (size_t)L.inner * sizeof(Acc);
    if (L.scratch_bytes < need || !L.scratch)
        return fail(TOMOS_ERR_INVALID,
                    "tomos_gemv: scratch too small (need " + std::to_string(need) + " bytes)");
    // few, long lines (a column-major A x): chunks of at least eight lines
    // until eight CTAs an SM, as far as the scratch holds their partials
    int64_t more = ((int64_t)sm_count() * 8 + xb - 1) / xb;
    if (more > (L.outer + 7) / 8) more = (L.outer + 7) / 8;
    const int64_t fit = (int64_t)(L.scratch_bytes / ((size_t)L.inner * sizeof(Acc)));
    if (more > fit) more = fit;
    if (more > nchunks) nchunks = more;
    const int64_t lpc = (L.outer + nchunks - 1) / nchunks;
    nchunks = (L.outer + lpc - 1) / lpc;
    dim3 grid((unsigned)xb, (unsigned)nchunks);
    Acc* partial = static_cast<Acc*>(L.scratch);
    line_sum_partial_kernel<E, ACC64, V><<<grid, 256, 0, st>>>(L.hi, L.lo, L.outer, L.inner, L.ld,
                                                               L.x, lpc, L.skip, partial);
    TOMOS_LAUNCH_CHECK("line_sum_partial_kernel");
    return sum_parts(partial, nchunks, L.inner, L.inner, L.alpha, L.beta, L.coef, L.skip, L.y, st);
}

// 16-byte loads where every line starts on a 16-byte boundary; sums of few
// lines (kVecSumLines) take an element a thread, which leaves more threads than
// a chunk each: 1e6 x 16 bf16, exact, 26 us in chunks, 18 us.
constexpr int64_t kVecSumLines = 128;

template <Elem E, bool ACC64>
static tomos_status run_gemv(const GemvLaunch& L, cudaStream_t st) {
    constexpr bool TWO = E == Elem::A16 || E == Elem::AB16 || E == Elem::AB16R;
    const int esz = E == Elem::F32 ? 4 : 2;
    const bool vec = (L.ld * esz) % 16 == 0 && reinterpret_cast<uintptr_t>(L.hi) % 16 == 0 &&
                     (!TWO || reinterpret_cast<uintptr_t>(L.lo) % 16 == 0) &&
                     (L.dot || L.outer >= kVecSumLines);
    return vec ? run_gemv_v<E, ACC64, ChunkElems<E>::value>(L, st) : run_gemv_v<E, ACC64, 1>(L, st);
}

template <Elem E>
static tomos_status run_gemv_acc(const GemvLaunch& L, bool acc64, cudaStream_t st) {
    return acc64 ? run_gemv<E, true>(L, st) : run_gemv<E, false>(L, st);
}

tomos_status gemv_launch(const GemvLaunch& L, Elem e, bool acc64, cudaStream_t st) {
    switch (e) {
        case Elem::F32: return run_gemv_acc<Elem::F32>(L, acc64, st);
        case Elem::H16: return run_gemv_acc<Elem::H16>(L, acc64, st);
        case Elem::F16: return run_gemv_acc<Elem::F16>(L, acc64, st);
        case Elem::A16: return run_gemv<Elem::A16, true>(L, st);
        case Elem::B16: return run_gemv_acc<Elem::B16>(L, acc64, st);
        case Elem::AB16: return run_gemv<Elem::AB16, true>(L, st);
        case Elem::AB16R: return run_gemv<Elem::AB16R, true>(L, st);
        default: return fail(TOMOS_ERR_UNSUPPORTED, "gemv: unsupported element type");
    }
}

bool elem_is_exact(Elem e) { return e == Elem::A16 || e == Elem::AB16 || e == Elem::AB16R; }

__global__ void scale_vec_kernel(float* y, int64_t n, double beta) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = beta != 0.0 ? (float)(beta * (double)y[i]) : 0.0f;
}

bool gemv_shape(const tomos_dense* A, int32_t trans, bool* dot, int64_t* outer, int64_t* inner,
                std::string* why) {
    if (!A) {
        *why = "null matrix";
        return false;
    }
    if (A->layout != TOMOS_ROW_MAJOR && A->layout != TOMOS_COL_MAJOR) {
        *why = "bad layout";
        return false;
    }
    if (trans != TOMOS_NO_TRANSPOSE && trans != TOMOS_TRANSPOSE) {
        *why = "bad transpose flag";
        return false;
    }
    if (A->rows < 0 || A->cols < 0) {
        *why = "negative dimension";
        return false;
    }
    bool row = A->layout == TOMOS_ROW_MAJOR;
    *outer = row ? A->rows : A->cols;
    *inner = row ? A->cols : A->rows;
    if (A->ld < *inner || A->ld < 1) {
        *why = "leading dimension smaller than the contiguous extent";
        return false;
    }
    *dot = (row == (trans == TOMOS_NO_TRANSPOSE));
    return true;
}

size_t gemv_scratch_bytes_max(const tomos_dense* A, int32_t trans) {
    bool dot;
    int64_t outer, inner;
    std::string why;
    if (!gemv_shape(A, trans, &dot, &outer, &inner, &why)) return 0;
    if (dot) {
        const int64_t segs = line_dot_segments(outer, inner);
        return segs > 1 ? (size_t)segs * (size_t)outer * sizeof(double) : 0;
    }
    const size_t generic = (size_t)line_sum_chunks(outer) * (size_t)inner * 8;
    const size_t rowpass = rowpass_gemv_scratch_bytes(outer, inner);
    return generic > rowpass ? generic : rowpass;
}

tomos_status gemv_dispatch(int32_t trans, double alpha, const tomos_dense* A, int32_t tier,
                           const float* x, double beta, float* y, void* scratch,
                           size_t scratch_bytes, cudaStream_t st) {
    GemvLaunch L;
    std::string why;
    if (!gemv_shape(A, trans, &L.dot, &L.outer, &L.inner, &why))
        return fail(TOMOS_ERR_INVALID, "tomos_gemv: " + why);
    Elem e;
    if (!resolve_elem(A, tier, &e, &why)) return fail(TOMOS_ERR_UNSUPPORTED, "tomos_gemv: " + why);
    int64_t ylen = (trans == TOMOS_NO_TRANSPOSE) ? A->rows : A->cols;
    if (ylen == 0) return TOMOS_OK;
    if (!y) return fail(TOMOS_ERR_INVALID, "tomos_gemv: null y");
    int64_t xlen = (trans == TOMOS_NO_TRANSPOSE) ? A->cols : A->rows;
    if (xlen == 0) {
        scale_vec_kernel<<<(unsigned)((ylen + 255) / 256), 256, 0, st>>>(y, ylen, beta);
        TOMOS_LAUNCH_CHECK("scale_vec_kernel");
        return TOMOS_OK;
    }
    if (!x || !A->values) return fail(TOMOS_ERR_INVALID, "tomos_gemv: null pointer");
    L.hi = A->values;
    L.lo = elem_is_exact(e) ? dense_lo_plane(A) : nullptr;
    L.ld = A->ld;
    L.x = x;
    L.y = y;
    L.alpha = alpha;
    L.beta = beta;
    L.scratch = scratch;
    L.scratch_bytes = scratch_bytes;
    bool used = false;
    tomos_status rs = rowpass_gemv(L, e, st, &used);
    if (used) return rs;
    return gemv_launch(L, e, elem_is_exact(e), st);
}

// Fixed scratch for tomos_gemv_no_alloc: the per-chunk partials of a
// line-sum product live in this module-scope buffer instead of caller
// memory.  The line-sum kernel writes every partial it later reduces, so
// nothing in it has to start at zero.
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;
constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) double g_gemv_static_scratch[kNoAllocScratchBytes / sizeof(double)];

// Device address of g_gemv_static_scratch on the current device, looked up
// on the first call made with that device current and cached afterwards.
static tomos_status no_alloc_scratch(void** out) {
    static std::mutex mu;
    static void* addr[kNoAllocMaxDevices] = {};
    int dev = 0;
    TOMOS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return fail(TOMOS_ERR_UNSUPPORTED, "tomos_gemv_no_alloc: device ordinal " +
                                               std::to_string(dev) + " out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_gemv_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(gemv static scratch)");
        addr[dev] = p;
    }
    *out = addr[dev];
    return TOMOS_OK;
}

tomos_status gemv_no_alloc(int32_t trans, double alpha, const tomos_dense* A, int32_t tier,
                           const float* x, double beta, float* y, cudaStream_t st) {
    const size_t need = gemv_scratch_bytes_max(A, trans);
    if (need > kNoAllocScratchBytes)
        return fail(TOMOS_ERR_INVALID,
                    "tomos_gemv_no_alloc: this product needs " + std::to_string(need) +
                        " bytes of scratch; the fixed buffer holds " +
                        std::to_string(kNoAllocScratchBytes) + " (use tomos_gemv)");
    void* scratch = nullptr;
    tomos_status s = no_alloc_scratch(&scratch);
    if (s) return s;
    return gemv_dispatch(trans, alpha, A, tier, x, beta, y, scratch, kNoAllocScratchBytes, st);
}

}  // namespace tomos_b200

using namespace tomos_b200;

extern "C" {

tomos_status tomos_gemv_no_alloc(int32_t trans, double alpha, const tomos_dense* A, int32_t tier,
                                 const float* x, double beta, float* y, void* stream) {
    return gemv_no_alloc(trans, alpha, A, tier, x, beta, y, as_stream(stream));
}

size_t tomos_gemv_scratch_bytes(const tomos_dense* A, int32_t trans) {
    // Sized for the widest (FP64-accumulating) tier so one buffer serves all.
    return gemv_scratch_bytes_max(A, trans);
}

tomos_status tomos_gemv(int32_t trans, double alpha, const tomos_dense* A, int32_t tier,
                        const float* x, double beta, float* y, void* scratch,
                        size_t scratch_bytes, void* stream) {
    return gemv_dispatch(trans, alpha, A, tier, x, beta, y, scratch, scratch_bytes,
                         as_stream(stream));
}

}  // extern "C"
