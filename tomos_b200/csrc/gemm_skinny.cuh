// gemm_skinny.cuh -- products C = alpha op(A) op(B) + beta C with at most 16
// columns and A read exactly (FP32 storage, or both planes of packed
// storage): three TF32 products of split operands, as kTf32x3, fed from
// registers.
//
// With so few columns the product is one pass over A, 0.6 ms of HBM time at
// 1e6 x 1000 FP32_16.  The tcgen05 pipeline decodes, splits and stores every
// element of A to shared memory as two TF32 tiles and was bound by that:
// 2.3 ms.  FP32 FMAs from registers were bound by the shuffles that add the
// lanes' sums (1.9 ms).  Here the fragments of mma.m16n8k8 are loaded from
// global memory as they lie: the order of K, and of the columns of A^T, is
// free, so a lane takes eight neighbouring elements of a line (16 bytes a
// plane) and the steps of a product take them two by two:
//   lines along K (skinny_dot_kernel)  a warp takes 16 lines x 32 K at a
//       time; op(B) is split once a CTA into shared memory, in fragment
//       order;
//   lines along M (skinny_sum_kernel)  a warp takes 64 columns of 8 lines at
//       a time, and the lines' part of op(B) from global memory; every warp
//       is on its own and writes one run's partial sums.
// What is left an element is its decode and its split.  No barrier and no
// shared-memory write in either loop; the next chunk is in
// flight in a warp's registers, later ones are asked into L2.
// 1e6 x 1000 x 16 FP32_16: 1.05 ms along K, 1.40 ms along M (3.8 and 2.9 TB/s;
// bound by the decode, the split and the products' issue together); 200000 x
// 500 x 8 FP32, both: 390 us to 217 us; unaligned 300000 x 257 x 16 FP32:
// 1.30 ms to 0.25 ms.
// Accuracy: the hardware's adds round toward zero, so a hardware sum is short:
// along K the products of 32 K, those with a small half apart, added to an
// FP32 total (48 adds at most); along M 48 lines, added to an FP64 total (a
// run of 16384 lines, as of the diagonal of A^T A, all of one sign).  Runs
// are summed in FP64 by the caller.  Relative to FP64: 1.7e-7 along K, 4e-7
// along M at 1e6 x 1000 (the tiled kernels 7e-6 and 4.6e-6); 1.0e-7 at K = 9
// and 16 (2.0e-7).
#pragma once

#include "common.cuh"
#include "fused.cuh"

namespace tomos_b200 {

struct SkinnyArgs {
    const void* hi;
    const void* lo;
    int64_t stride;    // elements between lines of A
    const float* b;
    int64_t b_sl, b_sj;  // op(B)(l, j) is element l b_sl + j b_sj
    float* c;
    int64_t c_si, c_sj;
    int64_t M, N, K;
    int64_t run;       // K of one run
    int runs;
    double alpha, beta;
    float* part;       // [run][N][M] FP32 sums (NULL: write C)
};

constexpr int kSkinnyMaxN = 16;
constexpr int kSkinnyDotWarps = 16;
constexpr int kSkinnyDotK = 1536;      // K of a run of skinny_dot_kernel: 192 KB of split op(B) at 16 columns
constexpr int kSkinnySumWarps = 4;
constexpr int kSkinnySumCtas = 3;      // an SM
constexpr int kSkinnySumLines = 16384; // lines of a run of skinny_sum_kernel, at most
constexpr int kSkinnyAhead = 8;        // chunks asked into L2 ahead

// x as two TF32 values, both rounded to nearest: 24 bits (truncated halves
// keep 22 and lean toward zero).  The first one's rounding is two integer
// instructions, cheaper than the conversion; a NaN whose carry leaves the
// exponent still has a NaN remainder.
__device__ __forceinline__ void skinny_split(float x, uint32_t& big, uint32_t& small) {
    big = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(small) : "f"(x - __uint_as_float(big)));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Eight elements of a line, raw: lane x of the W lanes that share the line's
// 8 W elements.  VECL: lines start on 16 bytes (both planes) and end on a
// whole 16-byte chunk; element by element otherwise.
template <Elem E, int W, bool VECL>
struct SkinnyWords {
    static constexpr bool F32 = E == Elem::F32;
    static constexpr int ESZ = F32 ? 4 : 2;
    uint32_t h[F32 ? 8 : 4], l[F32 ? 1 : 4];

    static __device__ __forceinline__ int elem(int x, int q) {
        if constexpr (!VECL) return q * W + x;
        else if constexpr (F32) return (q >> 2) * (4 * W) + 4 * x + (q & 3);
        else return 8 * x + q;
    }
    // elements elem(x, q) < left of the part of a line at `hi` (its other
    // plane `lo` bytes further); zeros elsewhere
    __device__ __forceinline__ void load(const uint8_t* hi, int64_t lo, bool in, int64_t left, int x) {
#pragma unroll
        for (int k = 0; k < (F32 ? 8 : 4); ++k) h[k] = 0u;
#pragma unroll
        for (int k = 0; k < (F32 ? 1 : 4); ++k) l[k] = 0u;
        if constexpr (VECL) {
            constexpr int V = F32 ? 4 : 8;
#pragma unroll
            for (int c = 0; c < 8 / V; ++c) {
                const int e = elem(x, c * V);
                if (in && e < left) {
                    const uint4 t = __ldcs(reinterpret_cast<const uint4*>(hi + e * ESZ));
                    h[4 * c] = t.x, h[4 * c + 1] = t.y, h[4 * c + 2] = t.z, h[4 * c + 3] = t.w;
                    if constexpr (!F32) {
                        const uint4 r = __ldcs(reinterpret_cast<const uint4*>(hi + lo + e * ESZ));
                        l[0] = r.x, l[1] = r.y, l[2] = r.z, l[3] = r.w;
                    }
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int e = elem(x, q);
                if (in && e < left) {
                    if constexpr (F32) {
                        h[q] = __ldg(reinterpret_cast<const uint32_t*>(hi + e * ESZ));
                    } else {
                        h[q >> 1] |= (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(hi + e * ESZ)) << (16 * (q & 1));
                        l[q >> 1] |= (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(hi + lo + e * ESZ)) << (16 * (q & 1));
                    }
                }
            }
        }
    }
    // elements 2 s and 2 s + 1
    __device__ __forceinline__ float2 pair(int s) const {
        if constexpr (F32) {
            return make_float2(__uint_as_float(h[2 * s]), __uint_as_float(h[2 * s + 1]));
        } else if constexpr (E == Elem::A16) {
            float2 v = decode_pair_fp32_16(h[s], l[s]);
            if (h[s] & 0x00010001u) v = decode_pair_fp32_16_exact(h[s], l[s]);
            return v;
        } else {
            return make_float2(word_value<E>(h[s] & 0xFFFFu, l[s] & 0xFFFFu), word_value<E>(h[s] >> 16, l[s] >> 16));
        }
    }
};

__device__ __forceinline__ void skinny_store(const SkinnyArgs& g, int64_t run, int64_t i, int64_t j, float v) {
    if (i >= g.M || j >= g.N) return;
    if (g.part) {
        g.part[(size_t)run * (size_t)g.M * (size_t)g.N + (size_t)(j * g.M + i)] = v;
        return;
    }
    float* cp = g.c + (size_t)(i * g.c_si + j * g.c_sj);
    double y = g.alpha * (double)v;
    if (g.beta != 0.0) y += g.beta * (double)*cp;
    *cp = (float)y;
}

// Lines along K.  blockIdx.y: the run; a warp walks tiles of 16 lines, each
// over the whole run.  NT: groups of 8 columns.
template <Elem E, int NT, bool VECL>
__global__ void __launch_bounds__(32 * kSkinnyDotWarps, 1) skinny_dot_kernel(SkinnyArgs g) {
    using Words = SkinnyWords<E, 4, VECL>;
    extern __shared__ __align__(16) float4 bs[];  // [chunk][step][column group][lane]: big, big, small, small
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 3, q8 = lane >> 2;
    const int64_t k0 = (int64_t)blockIdx.y * g.run;
    const int64_t k1 = k0 + g.run < g.K ? k0 + g.run : g.K;
    const int nc = (int)((k1 - k0 + 31) / 32);
    for (int i = threadIdx.x; i < nc * 4 * NT * 32; i += blockDim.x) {
        const int l = i & 31, j = (i >> 5) % NT, cs = (i >> 5) / NT;
        const int64_t col = 8 * j + (l >> 2);
        uint32_t bg[2], sm[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t k = k0 + (cs >> 2) * 32 + Words::elem(l & 3, 2 * (cs & 3) + e);
            skinny_split((k < k1 && col < g.N) ? __ldg(g.b + (k * g.b_sl + col * g.b_sj)) : 0.0f, bg[e], sm[e]);
        }
        bs[i] = make_float4(__uint_as_float(bg[0]), __uint_as_float(bg[1]), __uint_as_float(sm[0]),
                            __uint_as_float(sm[1]));
    }
    __syncthreads();
    const int64_t tiles = (g.M + 15) / 16, step = (int64_t)gridDim.x * kSkinnyDotWarps;
    int64_t tile = (int64_t)warp * gridDim.x + blockIdx.x;
    int c = 0;
    int64_t ltile = tile;  // the next chunk to load
    int lc = 0;
    Words w[2][2];
    const int64_t pitch = g.stride * Words::ESZ;
    const int64_t lo = static_cast<const uint8_t*>(g.lo) - static_cast<const uint8_t*>(g.hi);
    const uint8_t* base = static_cast<const uint8_t*>(g.hi) + k0 * Words::ESZ;
    const uint8_t* line = base + (ltile * 16 + q8) * pitch;
    auto load = [&](Words (&d)[2]) {
        const int64_t i = ltile * 16 + q8, left = k1 - k0 - lc * 32;
        const uint8_t* at = line + lc * (32 * Words::ESZ);
        d[0].load(at, lo, i < g.M, left, t);
        d[1].load(at + 8 * pitch, lo, i + 8 < g.M, left, t);
        // two chunks' 128-byte lines (one chunk's of FP32) of this lane's line, ahead
        if (Words::F32 || (lc & 1) == 0) {
            const int pc = lc + kSkinnyAhead;
            const int64_t pi = ltile * 16 + (lane & 15);
            const uint8_t* pa = base + pi * pitch + pc * (32 * Words::ESZ);
            if (pc < nc && pi < g.M && (!Words::F32 || lane < 16)) prefetch_l2(lane < 16 ? pa : pa + lo);
        }
        if (++lc == nc) {
            lc = 0;
            ltile += step;
            line += step * 16 * pitch;
        }
    };
    load(w[0]);
    float tot[NT][4] = {};
    while (tile < tiles) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            load(w[u ^ 1]);
            float d[NT][4] = {}, ds[NT][4] = {};  // ds: the products with a small half
            const float4* bp = bs + (size_t)c * (4 * NT * 32) + lane;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float2 x0 = w[u][0].pair(s), x1 = w[u][1].pair(s);
                uint32_t bg[4], sm[4];
                skinny_split(x0.x, bg[0], sm[0]);
                skinny_split(x1.x, bg[1], sm[1]);
                skinny_split(x0.y, bg[2], sm[2]);
                skinny_split(x1.y, bg[3], sm[3]);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const float4 b = bp[(s * NT + j) * 32];
                    mma_tf32(ds[j], bg, __float_as_uint(b.z), __float_as_uint(b.w));
                    mma_tf32(ds[j], sm, __float_as_uint(b.x), __float_as_uint(b.y));
                    mma_tf32(d[j], bg, __float_as_uint(b.x), __float_as_uint(b.y));
                }
            }
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) tot[j][e] += d[j][e] + ds[j][e];
            if (++c == nc) {
                if (tile < tiles) {
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            skinny_store(g, blockIdx.y, tile * 16 + q8 + 8 * (e >> 1), 8 * j + 2 * t + (e & 1), tot[j][e]);
                            tot[j][e] = 0.0f;
                        }
                }
                c = 0;
                tile += step;
            }
        }
    }
}

// Lines along M.  A warp owns 64 columns of one run of lines.
template <Elem E, int NT, bool VECL>
__global__ void __launch_bounds__(32 * kSkinnySumWarps, kSkinnySumCtas) skinny_sum_kernel(SkinnyArgs g) {
    using Words = SkinnyWords<E, 8, VECL>;
    const int lane = threadIdx.x & 31, t = lane & 3, q8 = lane >> 2;
    const int64_t groups = (g.M + 63) / 64;
    const int64_t wid = (int64_t)blockIdx.x * kSkinnySumWarps + (threadIdx.x >> 5);
    const int64_t run = wid / groups, e0 = (wid % groups) * 64;
    if (run >= g.runs) return;
    const int64_t k0 = run * g.run;
    const int64_t k1 = k0 + g.run < g.K ? k0 + g.run : g.K;
    // the FP64 totals: 16 fit the registers, 32 would be spilled
    constexpr bool SM = NT > 1;
    __shared__ double tsum[SM ? kSkinnySumWarps : 1][SM ? 16 * NT : 1][32];
    double treg[SM ? 1 : 16];
    auto tot = [&](int p, int j, int e) -> double& {
        if constexpr (SM) return tsum[threadIdx.x >> 5][(p * NT + j) * 4 + e][lane];
        else return treg[p * 4 + e];
    };
#pragma unroll
    for (int i = 0; i < 16 * NT; ++i) tot(i / (4 * NT), i / 4 % NT, i % 4) = 0.0;
    Words w[2][2];
    float b[2][NT][2];
    const int64_t pitch = g.stride * Words::ESZ, left = g.M - e0;
    const int64_t lo = static_cast<const uint8_t*>(g.lo) - static_cast<const uint8_t*>(g.hi);
    int64_t lk = k0 + t;  // the next lines to load: lk and lk + 4
    const uint8_t* at = static_cast<const uint8_t*>(g.hi) + lk * pitch + e0 * Words::ESZ;
    const float* bp = g.b + lk * g.b_sl + q8 * g.b_sj;
    // lane: a 128-byte line of the 16 (8 lines of A, two planes or FP32 halves)
    const int64_t ahead = (int64_t)(8 * kSkinnyAhead + (lane & 7) - t) * pitch +
                          ((lane & 8) ? (Words::F32 ? (int64_t)128 : lo) : (int64_t)0);
    auto load = [&](Words (&d)[2], float (&x)[NT][2]) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const bool in = lk + 4 * e < k1;
            d[e].load(at + 4 * e * pitch, lo, in, left, q8);
#pragma unroll
            for (int j = 0; j < NT; ++j)
                x[j][e] = (in && 8 * j + q8 < g.N) ? __ldg(bp + 4 * e * g.b_sl + 8 * j * g.b_sj) : 0.0f;
        }
        if (lane < 16 && lk - t + 8 * kSkinnyAhead + 8 <= k1 && (!Words::F32 || lane < 8 || left > 32))
            prefetch_l2(at + ahead);
        lk += 8;
        at += 8 * pitch;
        bp += 8 * g.b_sl;
    };
    load(w[0], b[0]);
    float d[4][NT][4] = {};
    int held = 0;
    for (int64_t k = k0; k < k1; k += 16) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            load(w[u ^ 1], b[u ^ 1]);
            uint32_t bb[NT][2], bm[NT][2];
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) skinny_split(b[u][j][e], bb[j][e], bm[j][e]);
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const float2 x0 = w[u][0].pair(p), x1 = w[u][1].pair(p);
                uint32_t bg[4], sm[4];
                skinny_split(x0.x, bg[0], sm[0]);
                skinny_split(x0.y, bg[1], sm[1]);
                skinny_split(x1.x, bg[2], sm[2]);
                skinny_split(x1.y, bg[3], sm[3]);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    mma_tf32(d[p][j], bg, bm[j][0], bm[j][1]);
                    mma_tf32(d[p][j], sm, bb[j][0], bb[j][1]);
                    mma_tf32(d[p][j], bg, bb[j][0], bb[j][1]);
                }
            }
        }
        if (++held < 3 && k + 16 < k1) continue;  // 48 lines in one hardware sum
        held = 0;
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    tot(p, j, e) += (double)d[p][j][e];
                    d[p][j][e] = 0.0f;
                }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                skinny_store(g, run, e0 + Words::elem(q8, 2 * p + (e >> 1)), 8 * j + 2 * t + (e & 1),
                             (float)tot(p, j, e));
}

template <Elem E, int NT, bool VECL>
inline tomos_status launch_skinny_t(const SkinnyArgs& g, bool lines_k, cudaStream_t st) {
    if (lines_k) {
        const size_t smem = (size_t)((g.run < g.K ? g.run : g.K) + 31) / 32 * (4 * NT * 32) * sizeof(float4);
        auto kern = skinny_dot_kernel<E, NT, VECL>;
        TOMOS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int64_t gx = (g.M + 15) / 16, cap = (sm_count() + g.runs - 1) / g.runs;
        if (gx > cap) gx = cap;
        kern<<<dim3((unsigned)gx, (unsigned)g.runs), 32 * kSkinnyDotWarps, smem, st>>>(g);
    } else {
        const int64_t warps = (g.M + 63) / 64 * g.runs;
        skinny_sum_kernel<E, NT, VECL><<<(unsigned)((warps + kSkinnySumWarps - 1) / kSkinnySumWarps),
                                         32 * kSkinnySumWarps, 0, st>>>(g);
    }
    TOMOS_LAUNCH_CHECK("skinny product");
    return TOMOS_OK;
}

// lines_k: op(A)'s lines run along K.
template <Elem E>
inline tomos_status launch_skinny(const SkinnyArgs& g, bool lines_k, cudaStream_t st) {
    const bool vec = (g.stride * (E == Elem::F32 ? 4 : 2)) % 16 == 0 &&
                     (lines_k ? g.K : g.M) % (E == Elem::F32 ? 4 : 8) == 0 && reinterpret_cast<uintptr_t>(g.hi) % 16 == 0 &&
                     (E == Elem::F32 || reinterpret_cast<uintptr_t>(g.lo) % 16 == 0);
    if (g.N <= 8)
        return vec ? launch_skinny_t<E, 1, true>(g, lines_k, st) : launch_skinny_t<E, 1, false>(g, lines_k, st);
    return vec ? launch_skinny_t<E, 2, true>(g, lines_k, st) : launch_skinny_t<E, 2, false>(g, lines_k, st);
}

}  // namespace tomos_b200
