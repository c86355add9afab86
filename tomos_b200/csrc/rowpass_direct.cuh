// rowpass_direct.cuh -- the row pass without a shared-memory ring, for the
// rows rowpass.cuh and rowpass_mma.cuh do not serve well:
//   * narrow rows (at most 32 chunks of 16 bytes).  The ring passes give a
//     warp a row, or 32 rows a barrier round trip: at 1e6 x 64 bf16 the
//     tensor-core pass took 359 us for 128 MB, 1.7 us a stage of 4.6 KB;
//     this pass takes 31 us (4.1 TB/s);
//   * rows that do not start on a 16-byte boundary, which no bulk copy can
//     fetch: the two generic kernels and their reduction took 390 us an
//     LSQR pass at 150001 x 777 FP32 (466 MB, read twice); this pass takes
//     95 us (4.9 TB/s).
// Same arithmetic as rowpass.cuh: ut_i = cp (A p)_i + cu u_i, partials of
// A^T ut and of ||ut||^2, from one read of A.
//
// Every load is an aligned 16-byte chunk.  Rows that start at any element
// sit in the chunks at a shift that repeats every 2, 4 or 8 rows, and a warp
// takes rows of one residue only (row w + 8 t of its CTA), so its shift, and
// with it the column of every register, is fixed; the words of neighbouring
// rows in a row's first and last chunk are cleared.  Chunks that would reach
// outside A (its first and last rows) are read element by element.
//
// LPR lanes share a row, so a warp load covers 32 / LPR rows; lane `sub` of
// a row takes chunks sub, sub + LPR, .. (C of them), the columns of p and of
// the A^T ut accumulators it keeps in registers.  U such groups of rows are
// in flight a warp, the next ones loaded while the current are summed where
// the registers allow it; no barrier before the CTA's final reduction.  Bound
// by HBM; each value costs its share of a load, its decode and two FMAs, each
// row one FP64 update of ut, done by one lane for all the rows a warp holds.
//
// ACC64 (the accurate passes) forms every product of both sums in FP64 and
// leaves FP64 partials, as the generic kernels do.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "fused.cuh"

namespace tomos_b200 {

constexpr int kDirectWarps = 8;  // a multiple of the shift's period (at most 8 rows)
constexpr int64_t kDirectMaxCols = 1024;

struct DirectParams {
    FusedParams f;
    double* qpart64;   // ACC64 partials (gridDim.x x qstride)
    int dot;           // form A p (else ut = cu u)
    int axpy;          // accumulate A^T ut
    int write_u;
    int aligned;       // direct_aligned
};

// How a pass covers rows of n columns.
struct DirectShape {
    int lpr = 0;  // lanes per row; 0: not served
    int c = 0;    // chunks per lane
};

// Row groups in flight: about 32 values a lane (16 beside FP64 columns), at
// most 8, or 4 where a lane forms ut of several.
constexpr int direct_u(int per, int lpr, bool acc64) {
    const int u = (acc64 ? 16 : 32) / per, cap = lpr < 8 ? 4 : 8;
    return u < 1 ? 1 : (u < cap ? u : cap);
}
// Whether the next rows are loaded before the current ones are summed: not
// where a row alone takes a lane's registers.
constexpr bool direct_prefetch(int per, bool acc64) { return acc64 || per <= 20; }

template <Elem E>
struct DirectElem {
    static constexpr bool TWO = E == Elem::A16 || E == Elem::AB16 || E == Elem::AB16R;
    static constexpr int ESZ = E == Elem::F32 ? 4 : 2;
    static constexpr int VEC = ChunkElems<E>::value;
    // elements [idx, idx + VEC) of a plane as a chunk, those outside
    // [lo, hi) as zero words
    static __device__ __noinline__ uint4 slow(const void* plane, int64_t idx, int64_t lo, int64_t hi) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        for (int e = 0; e < VEC; ++e) {
            const int64_t k = idx + e;
            if (k < lo || k >= hi) continue;
            if constexpr (ESZ == 4) w[e] = __ldg(static_cast<const uint32_t*>(plane) + k);
            else w[e >> 1] |= (uint32_t)__ldg(static_cast<const uint16_t*>(plane) + k) << (16 * (e & 1));
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
    static __device__ __forceinline__ uint4 chunk(const void* plane, int64_t idx) {
        return __ldg(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(plane) + idx * ESZ));
    }
    static __device__ __forceinline__ void decode(uint4 h, const uint4& l, float* v) {
        if constexpr (E == Elem::H16) {
            if ((h.x | h.y | h.z | h.w) & 0x00010001u) fix_half_chunk(h);
            ChunkDecoder<Elem::F16>::decode(h, l, v);
        } else {
            ChunkDecoder<E>::decode(h, l, v);
        }
    }
};

template <Elem E, int LPR, int C, bool ACC64>
__global__ void __launch_bounds__(kDirectWarps * 32, ACC64 && C * ChunkElems<E>::value > 12 ? 1 : 2)
fused_direct_kernel(DirectParams T) {
    const FusedParams& P = T.f;
    if (P.skip && *P.skip) return;
    using D = DirectElem<E>;
    using Acc = typename std::conditional<ACC64, double, float>::type;
    constexpr int VEC = D::VEC, PER = VEC * C, U = direct_u(PER, LPR, ACC64), GR = 32 / LPR, RPS = GR * U;
    constexpr int K = (U + LPR - 1) / LPR;  // rows whose ut a lane forms
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ double ssw[kDirectWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane % LPR, grp = lane / LPR;
    const double cp = P.coef ? P.coef[0] : P.cp;
    const double cu = P.coef ? P.coef[1] : P.cu;
    const bool dot = T.dot != 0, axpy = T.axpy != 0;
    const bool use_u = P.coef || cu != 0.0;  // a product with cu == 0 never reads u
    const int n = (int)P.n;

    // the CTA's rows; row (u, grp) of iteration t is r0 + warp rw + grp rg + u ru + t ri
    const int64_t per = ((P.m + gridDim.x - 1) / gridDim.x + 7) / 8 * 8;
    const int64_t r0 = (int64_t)blockIdx.x * per;
    const int64_t r1 = r0 + per < P.m ? r0 + per : P.m;
    const int rows = r1 > r0 ? (int)(r1 - r0) : 0;
    const int rw = T.aligned ? RPS : 1, rg = T.aligned ? 1 : 8, ru = T.aligned ? GR : 8 * GR;
    constexpr int ri = kDirectWarps * RPS;
    // elements between the chunk boundary at or before a row's start and it
    const int shift =
        T.aligned ? 0
                  : (int)(((reinterpret_cast<uintptr_t>(P.hi) + (uintptr_t)((r0 + warp) * P.ld) * D::ESZ) % 16) / D::ESZ);
    // elements a chunk may touch, and the chunks of a row
    const int64_t lim = T.aligned ? P.m * P.ld : (P.m - 1) * P.ld + n;
    const int nch = (n + shift + VEC - 1) / VEC;

    // element e of chunk c of this lane is column (c LPR + sub) VEC + e - shift
    Acc pv[PER], acc[PER];
    uint32_t mask = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int col = ((j / VEC) * LPR + sub) * VEC + j % VEC - shift;
        const bool in = col >= 0 && col < n;
        if (in) mask |= 1u << j;
        pv[j] = (dot && in) ? (Acc)__ldg(P.p + col) : (Acc)0;
        acc[j] = (Acc)0;
    }
    // A row's first chunk may hold words of the row before (shift > 0), its
    // last one words past column n, neighbours or padding of any bits: those
    // are cleared in the loaded words.  What a cleared word decodes to is
    // finite, meets a zero of p, and adds to an accumulator nobody reads.
    const int clast = (nch - 1) / LPR;
    const bool efirst = shift > 0, elast = (n + shift) % VEC != 0;
    auto word_mask = [&](int ch) {
        uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            const int col = ch * VEC + e - shift;
            if (col >= 0 && col < n) m[e * D::ESZ / 4] |= D::ESZ == 4 ? 0xffffffffu : 0xffffu << (16 * (e & 1));
        }
        return make_uint4(m[0], m[1], m[2], m[3]);
    };
    const uint4 mfirst = word_mask(sub), mlast = word_mask(clast * LPR + sub);
    auto clear = [](uint4& x, const uint4& m) {
        x.x &= m.x;
        x.y &= m.y;
        x.z &= m.z;
        x.w &= m.w;
    };
    double ss = 0.0;
    const float* uip = P.u_in + r0;
    float* uop = P.u_out + r0;

    uint4 h[U][C], l[D::TWO ? U : 1][D::TWO ? C : 1];
    float uin[K];
    auto load = [&](int b) {  // the rows of the iteration whose first row is r0 + b
        const int64_t first = (r0 + b) * P.ld - shift;
        int64_t last = r0 + b + (int64_t)(GR - 1) * rg + (int64_t)(U - 1) * ru;
        // narrow rows, many a batch: those past A are not read, and aligned
        // ones never reach past it
        if (C == 1 && last >= P.m) last = P.m - 1;
        last = last * P.ld - shift + (int64_t)nch * VEC;
        // one branch for the whole batch: inside it the loads are predicated
        // only, so all of them issue before the first is waited for
        if ((C == 1 && T.aligned) || (first >= 0 && last <= lim)) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = b + grp * rg + u * ru;
                const int64_t idx = (r0 + i) * P.ld - shift;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int ch = c * LPR + sub;
                    h[u][c] = make_uint4(0u, 0u, 0u, 0u);
                    if constexpr (D::TWO) l[u][c] = make_uint4(0u, 0u, 0u, 0u);
                    if (i < rows && ch < nch) {
                        h[u][c] = D::chunk(P.hi, idx + (int64_t)ch * VEC);
                        if constexpr (D::TWO) l[u][c] = D::chunk(P.lo, idx + (int64_t)ch * VEC);
                    }
                }
            }
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = b + grp * rg + u * ru;
                const int64_t idx = (r0 + i) * P.ld - shift;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int ch = c * LPR + sub;
                    const bool in = i < rows && ch < nch;
                    const int64_t at = idx + (int64_t)ch * VEC;
                    if (C == 1 && in && at >= 0 && at + VEC <= lim) {
                        h[u][c] = D::chunk(P.hi, at);
                        if constexpr (D::TWO) l[u][c] = D::chunk(P.lo, at);
                        continue;
                    }
                    if (C == 1 && !in) {
                        h[u][c] = make_uint4(0u, 0u, 0u, 0u);
                        if constexpr (D::TWO) l[u][c] = make_uint4(0u, 0u, 0u, 0u);
                        continue;
                    }
                    h[u][c] = D::slow(P.hi, at, 0, in ? lim : 0);
                    if constexpr (D::TWO) l[u][c] = D::slow(P.lo, at, 0, in ? lim : 0);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int i = b + grp * rg + (sub + q * LPR) * ru;
            uin[q] = (use_u && sub + q * LPR < U && i < rows) ? __ldg(uip + i) : 0.0f;
        }
    };
    constexpr bool PRE = direct_prefetch(PER, ACC64);
    if (PRE) load(warp * rw);
    for (int b = warp * rw; b < rows; b += ri) {
        float v[U][PER], ur[K], ut[U];
        Acc d[U];
        if (!PRE) {
            // no registers for the next row: its lines (one a lane) go to L2
            // two rounds ahead
            const int64_t next = (int64_t)b + 2 * ri, off = (int64_t)lane * 128;
            if (next < rows && off < (int64_t)n * D::ESZ) {
                const size_t at = (size_t)(r0 + next) * P.ld * D::ESZ + off;
                prefetch_l2(static_cast<const uint8_t*>(P.hi) + at);
                if constexpr (D::TWO) prefetch_l2(static_cast<const uint8_t*>(P.lo) + at);
            }
        }
        if (!PRE) load(b);
        if (efirst) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                clear(h[u][0], mfirst);
                if constexpr (D::TWO) clear(l[u][0], mfirst);
            }
        }
        if (elast) {
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (c == clast) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        clear(h[u][c], mlast);
                        if constexpr (D::TWO) clear(l[u][c], mlast);
                    }
                }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < C; ++c) D::decode(h[u][c], l[D::TWO ? u : 0][D::TWO ? c : 0], &v[u][c * VEC]);
#pragma unroll
        for (int q = 0; q < K; ++q) ur[q] = uin[q];
        if (PRE) load(b + ri);
        if (dot) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (ACC64) {
                    Acc d0 = (Acc)0, d1 = (Acc)0;
#pragma unroll
                    for (int j = 0; j < PER; j += 2) {
                        d0 = fma((Acc)v[u][j], pv[j], d0);
                        d1 = fma((Acc)v[u][j + 1], pv[j + 1], d1);
                    }
                    d[u] = d0 + d1;
                } else {
                    float2 d0 = make_float2(0.0f, 0.0f), d1 = d0;
#pragma unroll
                    for (int j = 0; j < PER; j += 4) {
                        d0 = __ffma2_rn(make_float2(v[u][j], v[u][j + 1]), make_float2(pv[j], pv[j + 1]), d0);
                        d1 = __ffma2_rn(make_float2(v[u][j + 2], v[u][j + 3]), make_float2(pv[j + 2], pv[j + 3]), d1);
                    }
                    d[u] = (d0.x + d1.x) + (d0.y + d1.y);
                }
            }
#pragma unroll
            for (int o = LPR >> 1; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < U; ++u) d[u] += __shfl_xor_sync(0xffffffffu, d[u], o);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) d[u] = (Acc)0;
        }
        // lane sub of a row group forms ut of its groups u = sub, sub + LPR, ..
#pragma unroll
        for (int q = 0; q < K; ++q) {
            Acc dq = d[0];
#pragma unroll
            for (int u = 1; u < U; ++u)
                if (sub + q * LPR == u) dq = d[u];
            const int i = b + grp * rg + (sub + q * LPR) * ru;
            const bool has = sub + q * LPR < U && i < rows;
            const double r = (dot ? cp * (double)dq : 0.0) + (use_u ? cu * (double)ur[q] : 0.0);
            ur[q] = has ? (float)r : 0.0f;
            if (has) {
                if (T.write_u) uop[i] = ur[q];
                ss += (double)ur[q] * (double)ur[q];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) ut[u] = __shfl_sync(0xffffffffu, ur[u / LPR], grp * LPR + u % LPR);
        if (axpy) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (ACC64) {
#pragma unroll
                    for (int j = 0; j < PER; ++j) acc[j] = fma((Acc)v[u][j], (Acc)ut[u], acc[j]);
                } else {
                    const float2 u2 = make_float2(ut[u], ut[u]);
#pragma unroll
                    for (int j = 0; j < PER; j += 2) {
                        const float2 s = __ffma2_rn(make_float2(v[u][j], v[u][j + 1]), u2, make_float2(acc[j], acc[j + 1]));
                        acc[j] = s.x;
                        acc[j + 1] = s.y;
                    }
                }
            }
        }
    }

    if (P.sspart) {
        ss = warp_sum(ss);
        if (lane == 0) ssw[warp] = ss;
    }
    if (axpy) {
        // the row groups of a warp, then the warps, in a fixed order
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
            for (int j = 0; j < PER; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
        Acc* red = reinterpret_cast<Acc*>(dsm);  // one row of LPR PER + VEC columns a warp
        if (grp == 0) {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int col = ((j / VEC) * LPR + sub) * VEC + j % VEC - shift;
                if ((mask >> j) & 1u) red[(size_t)warp * (LPR * PER) + col] = acc[j];
            }
        }
    }
    __syncthreads();
    if (axpy) {
        const Acc* red = reinterpret_cast<const Acc*>(dsm);
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kDirectWarps; ++w) s += (double)red[(size_t)w * (LPR * PER) + j];
            if constexpr (ACC64)
                T.qpart64[(size_t)blockIdx.x * P.qstride + j] = s;
            else
                P.qpart[(size_t)blockIdx.x * P.qstride + j] = (float)s;
        }
    }
    if (P.sspart && threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kDirectWarps; ++w) s += ssw[w];
        P.sspart[blockIdx.x] = s;
    }
}

// Whether every row starts on a 16-byte boundary (both planes of two-plane
// types); P.ld, hi and lo as in FusedParams.
inline bool direct_aligned(Elem e, int64_t ld, const void* hi, const void* lo) {
    const bool two = e == Elem::A16 || e == Elem::AB16 || e == Elem::AB16R;
    return (ld * (e == Elem::F32 ? 4 : 2)) % 16 == 0 && reinterpret_cast<uintptr_t>(hi) % 16 == 0 &&
           (!two || reinterpret_cast<uintptr_t>(lo) % 16 == 0);
}

// The pass over rows of n columns at leading dimension ld: aligned rows of
// at most 32 chunks (wider ones run at the HBM rate in the ring passes), and
// unaligned rows of up to 32 values a lane (1021 FP32 or 1017 16-bit
// columns) whose planes have the same shift.
inline DirectShape direct_shape(Elem e, int64_t n, int64_t ld, const void* hi, const void* lo) {
    DirectShape s;
    if (e == Elem::F64 || n <= 0) return s;
    const bool two = e == Elem::A16 || e == Elem::AB16 || e == Elem::AB16R;
    const int esz = e == Elem::F32 ? 4 : 2, vec = 16 / esz;
    const bool aligned = direct_aligned(e, ld, hi, lo);
    if (!aligned) {
        if (reinterpret_cast<uintptr_t>(hi) % esz != 0 ||
            (two && reinterpret_cast<uintptr_t>(lo) % 16 != reinterpret_cast<uintptr_t>(hi) % 16))
            return s;
    }
    const int64_t nch = aligned ? (n + vec - 1) / vec : (n + 2 * vec - 2) / vec;  // at any shift
    if (nch <= 32) {
        s.c = 1;
        s.lpr = 2;
        while (s.lpr < nch) s.lpr *= 2;
    } else if (!aligned && nch <= 32 * (32 / vec)) {
        s.lpr = 32;
        s.c = (int)((nch + 31) / 32);
    }
    return s;
}

// CTAs: two an SM, at least 16 rows each (the latency of small products).
inline int direct_grid(int64_t m) {
    int64_t g = (int64_t)sm_count() * 2;
    if (g > (m + 15) / 16) g = (m + 15) / 16;
    return g < 1 ? 1 : (int)g;
}

template <Elem E, bool ACC64, int LPR, int C>
inline tomos_status launch_direct_t(const DirectParams& P, int grid, cudaStream_t st) {
    const size_t smem = P.axpy ? (size_t)kDirectWarps * LPR * C * ChunkElems<E>::value * (ACC64 ? 8 : 4) : 0;
    auto kern = fused_direct_kernel<E, LPR, C, ACC64>;
    if (smem > 40 * 1024)  // 48 KB with the static part
        TOMOS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, kDirectWarps * 32, smem, st>>>(P);
    TOMOS_LAUNCH_CHECK("fused_direct_kernel");
    return TOMOS_OK;
}

template <Elem E, bool ACC64>
inline tomos_status launch_direct_e(const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st) {
    if (s.lpr < 32) {
        switch (s.lpr) {
            case 2: return launch_direct_t<E, ACC64, 2, 1>(P, grid, st);
            case 4: return launch_direct_t<E, ACC64, 4, 1>(P, grid, st);
            case 8: return launch_direct_t<E, ACC64, 8, 1>(P, grid, st);
            case 16: return launch_direct_t<E, ACC64, 16, 1>(P, grid, st);
            default: break;
        }
    } else {
        switch (s.c) {
            case 1: return launch_direct_t<E, ACC64, 32, 1>(P, grid, st);
            case 2: return launch_direct_t<E, ACC64, 32, 2>(P, grid, st);
            case 3: return launch_direct_t<E, ACC64, 32, 3>(P, grid, st);
            case 4: return launch_direct_t<E, ACC64, 32, 4>(P, grid, st);
            default: break;
        }
        if constexpr (E == Elem::F32) {
            switch (s.c) {
                case 5: return launch_direct_t<E, ACC64, 32, 5>(P, grid, st);
                case 6: return launch_direct_t<E, ACC64, 32, 6>(P, grid, st);
                case 7: return launch_direct_t<E, ACC64, 32, 7>(P, grid, st);
                case 8: return launch_direct_t<E, ACC64, 32, 8>(P, grid, st);
                default: break;
            }
        }
    }
    return fail(TOMOS_ERR_UNSUPPORTED, "direct pass: no instantiation");
}

// One translation unit per storage family instantiates the kernels.
tomos_status launch_direct_f32(bool acc64, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st);
tomos_status launch_direct_half(Elem e, bool acc64, const DirectParams& P, const DirectShape& s, int grid,
                                cudaStream_t st);
tomos_status launch_direct_bf16(bool acc64, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st);
tomos_status launch_direct_exact(Elem e, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st);

inline tomos_status launch_direct(Elem e, bool acc64, const DirectParams& P, const DirectShape& s, int grid,
                                  cudaStream_t st) {
    switch (e) {
        case Elem::F32: return launch_direct_f32(acc64, P, s, grid, st);
        case Elem::H16:
        case Elem::F16: return launch_direct_half(e, acc64, P, s, grid, st);
        case Elem::B16: return launch_direct_bf16(acc64, P, s, grid, st);
        case Elem::A16:
        case Elem::AB16:
        case Elem::AB16R: return launch_direct_exact(e, P, s, grid, st);
        default: return fail(TOMOS_ERR_UNSUPPORTED, "direct pass: element type");
    }
}

}  // namespace tomos_b200
