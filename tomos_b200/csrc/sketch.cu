// sketch.cu -- hash CountSketch SA = S A (tomos_countsketch_*).
//
// S is the reference's hash sketch (countsketch_kernels.cpp:59-85,
// countsketch_cuda_kernels.cu:267-286): row i of A is added, with sign
// +1 if bit 0 of splitmix64(i ^ sign_seed) is set and -1 otherwise, into
// row splitmix64(i ^ bucket_seed) mod s of SA.  Integer hashing is
// bit-exact with the reference.  Unlike the reference (atomicAdd scatter,
// order-dependent float sums), every bucket here is summed by one owner in
// a fixed order, so SA is deterministic: row-major matrices in FP32, as the
// reference's sums, column-major and CSR ones in FP64.
//   1. per row segment: hash, and the segment's count of every bucket
//   2. exclusive scans: over the segments of a bucket, then over buckets
//   3. each segment places its rows in order: a stable counting sort, so a
//      bucket lists its rows ascending (bit 31 of an entry: sign -1)
//   4. owner sums        (row-major: threads own columns and walk the
//                         bucket's rows; column-major: a warp per (column,
//                         bucket) gathers down a contiguous column)
// More buckets than a segment's shared counters hold (kCsMaxCounted) take a
// global histogram, an unordered scatter and a sort of each bucket instead.
// The sum of squares of the values read (||A||_F^2) falls out of step 4.
#include <string>

#include "common.cuh"
#include "fused.cuh"
#include "mbarrier.cuh"  // smem_addr
#include "sketch.cuh"

namespace tomos_b200 {

// Row i of this matrix is row row0 + i of the whole problem (a row shard);
// the hash takes the whole problem's row index.
__global__ void cs_hash_kernel(int64_t m, int64_t s, uint64_t bseed, uint64_t sseed, int64_t row0,
                               int32_t* __restrict__ bucket, int8_t* __restrict__ sign,
                               int32_t* __restrict__ counts) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t gi = (uint64_t)(row0 + i);
        const int32_t b = (int32_t)(splitmix64(gi ^ bseed) % (uint64_t)s);
        bucket[i] = b;
        sign[i] = (splitmix64(gi ^ sseed) & 1ull) ? (int8_t)1 : (int8_t)-1;
        if (counts) atomicAdd(&counts[b], 1);
    }
}

// Step 1: segment blockIdx.x hashes its rows (bucket[i], bit 31 set for
// sign -1) and counts its buckets in shared memory into cnt[segment][bucket].
__global__ void __launch_bounds__(256) cs_count_kernel(int64_t m, int64_t per, int32_t s, uint64_t bseed,
                                                       uint64_t sseed, int64_t row0,
                                                       uint32_t* __restrict__ bucket,
                                                       int32_t* __restrict__ cnt) {
    extern __shared__ int32_t hist[];
    for (int j = threadIdx.x; j < s; j += blockDim.x) hist[j] = 0;
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * per;
    const int64_t r1 = r0 + per < m ? r0 + per : m;
    for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
        const uint64_t gi = (uint64_t)(row0 + i);
        const uint32_t b = (uint32_t)(splitmix64(gi ^ bseed) % (uint64_t)s);
        bucket[i] = b | ((splitmix64(gi ^ sseed) & 1ull) ? 0u : kCsNeg);
        atomicAdd(&hist[b], 1);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < s; j += blockDim.x) cnt[(size_t)blockIdx.x * s + j] = hist[j];
}

// Step 2a: cnt[g][j] := rows of bucket j in the segments before g, tot[j] :=
// all of them.  A CTA owns 32 buckets; its 32 warps split the segments.
__global__ void __launch_bounds__(1024) cs_segment_scan_kernel(int32_t* __restrict__ cnt, int nseg, int32_t s,
                                                               int32_t* __restrict__ tot) {
    __shared__ int32_t part[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * 32 + lane;
    const int per = (nseg + 31) / 32;
    const int g0 = w * per < nseg ? w * per : nseg;
    const int g1 = g0 + per < nseg ? g0 + per : nseg;
    int32_t sum = 0;
    if (j < s) {
#pragma unroll 8
        for (int g = g0; g < g1; ++g) sum += cnt[(size_t)g * s + j];
    }
    part[w][lane] = sum;
    __syncthreads();
    int32_t run = 0;
    for (int h = 0; h < w; ++h) run += part[h][lane];
    if (j >= s) return;
    if (w == 31) tot[j] = run + sum;
    int g = g0;
    for (; g + 8 <= g1; g += 8) {
        int32_t c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) c[u] = cnt[(size_t)(g + u) * s + j];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            cnt[(size_t)(g + u) * s + j] = run;
            run += c[u];
        }
    }
    for (; g < g1; ++g) {
        const int32_t c = cnt[(size_t)g * s + j];
        cnt[(size_t)g * s + j] = run;
        run += c;
    }
}

// Step 3: segment blockIdx.x places its rows in increasing order.  Its
// buckets' cursors sit in shared memory; one warp takes 32 rows a step, rows
// of the same bucket ranked by lane (match_any), so the order is the rows'.
__global__ void __launch_bounds__(256) cs_place_kernel(int64_t m, int64_t per, int32_t s,
                                                       const uint32_t* __restrict__ bucket,
                                                       const int32_t* __restrict__ cnt,
                                                       const int32_t* __restrict__ offsets,
                                                       uint32_t* __restrict__ perm) {
    extern __shared__ int32_t cur[];
    for (int j = threadIdx.x; j < s; j += blockDim.x) cur[j] = offsets[j] + cnt[(size_t)blockIdx.x * s + j];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const int64_t r0 = (int64_t)blockIdx.x * per;
    const int64_t r1 = r0 + per < m ? r0 + per : m;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t next = r0 + lane < r1 ? bucket[r0 + lane] : 0u;
    for (int64_t i0 = r0; i0 < r1; i0 += 32) {
        const uint32_t e = next;
        const int64_t i = i0 + lane;
        if (i + 32 < r1) next = bucket[i + 32];
        const bool in = i < r1;
        // lanes past the segment's end form a group of their own
        const uint32_t b = in ? (e & ~kCsNeg) : 0xffffffffu;
        const uint32_t same = __match_any_sync(0xffffffffu, b);
        const int rank = __popc(same & below);
        int32_t base = 0;
        if (in) base = cur[b];
        __syncwarp();
        if (in) {
            if (rank == 0) cur[b] = base + __popc(same);
            perm[base + rank] = (uint32_t)i | (e & kCsNeg);
        }
        __syncwarp();
    }
}

// Exclusive scan of counts[0..s) into offsets[0..s], one block.
__global__ void cs_scan_kernel(const int32_t* __restrict__ counts, int64_t s,
                               int32_t* __restrict__ offsets) {
    __shared__ int32_t carry;
    __shared__ int32_t wsum[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t base = 0; base < s; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        int32_t v = i < s ? counts[i] : 0;
        int32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            int32_t t = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            wsum[lane] = t;
        }
        __syncthreads();
        const int32_t before = carry + (w > 0 ? wsum[w - 1] : 0) + x - v;
        if (i < s) offsets[i] = before;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = before + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) offsets[s] = carry;
}

__global__ void cs_scatter_kernel(int64_t m, const int32_t* __restrict__ bucket,
                                  const int8_t* __restrict__ sign, const int32_t* __restrict__ offsets,
                                  int32_t* __restrict__ cursor, uint32_t* __restrict__ perm) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t b = bucket[i];
        perm[offsets[b] + atomicAdd(&cursor[b], 1)] = (uint32_t)i | (sign[i] < 0 ? kCsNeg : 0u);
    }
}

// Sorts each bucket's row ids ascending, a warp per bucket (buckets hold
// about m/s rows): a bitonic network in shared memory for buckets of up to
// kCsSortCap rows, odd-even transposition in place for longer ones.
constexpr int kCsSortCap = 1024;
constexpr int kCsSortWarps = 4;

__global__ void __launch_bounds__(kCsSortWarps * 32) cs_sort_kernel(int64_t s,
                                                                  const int32_t* __restrict__ offsets,
                                                                  uint32_t* __restrict__ perm) {
    __shared__ uint32_t buf[kCsSortWarps][kCsSortCap];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t b = (int64_t)blockIdx.x * kCsSortWarps + w;
    if (b >= s) return;
    const int32_t o0 = offsets[b], len = offsets[b + 1] - o0;
    uint32_t* seg = perm + o0;
    if (len > kCsSortCap) {
        for (int32_t pass = 0; pass < len; ++pass) {
            const int32_t start = pass & 1;
            for (int32_t k = start + 2 * lane; k + 1 < len; k += 64) {
                const uint32_t x = seg[k], y = seg[k + 1];
                if ((x & ~kCsNeg) > (y & ~kCsNeg)) {
                    seg[k] = y;
                    seg[k + 1] = x;
                }
            }
            __syncwarp();
        }
        return;
    }
    int N = 1;
    while (N < len) N <<= 1;
    uint32_t* v = buf[w];
    for (int e = lane; e < N; e += 32) v[e] = e < len ? seg[e] : 0x7fffffff;
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            // pairs (i, i ^ j) with i < i ^ j are disjoint within a step
            for (int i = lane; i < N; i += 32) {
                const int p = i ^ j;
                if (p > i) {
                    const uint32_t x = v[i], y = v[p];
                    if (((x & ~kCsNeg) > (y & ~kCsNeg)) == ((i & k) == 0)) {
                        v[i] = y;
                        v[p] = x;
                    }
                }
            }
            __syncwarp();
        }
    }
    for (int e = lane; e < len; e += 32) seg[e] = v[e];
}

// Row-major owner sums.  Sums are FP32 with the rows of a bucket in
// increasing order, bit for bit the reference's countsketch_apply_impl<float>
// (countsketch_kernels.cpp:70-83); every bucket writes its row of SA and its
// FP32 column sums of squares (col_part, s x n), which cs_colsq_chunk_kernel
// reduces in bucket order.
//
// STAGE (FP32_16 HALF tier only): the fp32_16_half_only words of every chunk
// read are also written to `plane` (row pitch ld_plane halves) -- the fixed
// fp16 copy of the wh plane the LSQR HALF-tier iterations read -- so a solve
// that follows the sketch needs no staging pass of its own.
struct CsRowsArgs {
    const void* hi;
    const void* lo;
    int64_t n, ld, s;
    const int32_t* offsets;
    const uint32_t* perm;
    double* SA;
    int64_t ld_sa;
    float* col_part;  // s x n
    uint16_t* plane;
    int64_t ld_plane;
};

template <Elem E>
struct CsElem {
    static constexpr int VEC = ChunkElems<E>::value;
    static constexpr int ESZ = (E == Elem::F32) ? 4 : 2;
    static constexpr int PLANES = (E == Elem::A16 || E == Elem::AB16 || E == Elem::AB16R) ? 2 : 1;
};

// One 16-byte chunk as float pairs (STAGE: its fixed words to `stage`).
template <Elem E, bool STAGE>
__device__ __forceinline__ void cs_chunk_values(uint4& h, const uint4& l, uint16_t* stage,
                                                float2 (&v)[CsElem<E>::VEC / 2]) {
    if constexpr (E == Elem::H16) {
        fix_half_chunk(h);
        if constexpr (STAGE) *reinterpret_cast<uint4*>(stage) = h;
        v[0] = h2f2(h.x);
        v[1] = h2f2(h.y);
        v[2] = h2f2(h.z);
        v[3] = h2f2(h.w);
    } else {
        float f[CsElem<E>::VEC];
        ChunkDecoder<E>::decode(h, l, f);
#pragma unroll
        for (int e = 0; e < CsElem<E>::VEC / 2; ++e) v[e] = make_float2(f[2 * e], f[2 * e + 1]);
    }
}

// Rows 16-byte aligned: a CTA takes one bucket and blockDim.x chunks of its
// rows, a thread one chunk.  Bound by HBM latency: a thread keeps kCsDepth
// rows' loads in flight (16 bytes each), the row ids of the next batch
// loaded before the current one is summed.  Chunks past column n are not
// touched; the elements of the last chunk past n are summed and dropped.
// 1e6 x 1000 FP32_16 with the staged plane (2 GB read, 2 GB written): 889 us
// (4.5 TB/s) against 937 us for a shared-memory ring per warp.
constexpr int kCsDepth = 8;
constexpr int kCsThreads = 128;  // chunks (threads) a CTA at most

template <Elem E, bool STAGE>
__global__ void __launch_bounds__(kCsThreads) cs_rows_kernel(CsRowsArgs a) {
    static_assert(!STAGE || E == Elem::H16, "staging writes FP32_16 wh planes");
    constexpr int VEC = CsElem<E>::VEC, HV = VEC / 2, ESZ = CsElem<E>::ESZ, PLANES = CsElem<E>::PLANES;
    constexpr int D = PLANES == 2 ? kCsDepth / 2 : kCsDepth;
    const int64_t b = blockIdx.x;
    const int64_t c = (int64_t)blockIdx.y * blockDim.x + threadIdx.x;
    if (c * VEC >= a.n) return;
    const int32_t o0 = a.offsets[b], len = a.offsets[b + 1] - o0;
    const uint32_t* ids = a.perm + o0;
    const uint8_t* hp = static_cast<const uint8_t*>(a.hi) + c * 16;
    const uint8_t* lp = static_cast<const uint8_t*>(a.lo) + c * 16;
    const size_t pitch = (size_t)a.ld * ESZ;
    float2 acc[HV], csq[HV];
#pragma unroll
    for (int e = 0; e < HV; ++e) acc[e] = csq[e] = make_float2(0.0f, 0.0f);
    uint32_t nid[D];
#pragma unroll
    for (int u = 0; u < D; ++u) nid[u] = u < len ? __ldg(ids + u) : 0u;
    for (int32_t q = 0; q < len; q += D) {
        uint32_t id[D];
        uint4 h[D], l[PLANES == 2 ? D : 1];
#pragma unroll
        for (int u = 0; u < D; ++u) {
            id[u] = nid[u];
            if (q + u < len) {
                const size_t off = (size_t)(id[u] & ~kCsNeg) * pitch;
                h[u] = __ldcs(reinterpret_cast<const uint4*>(hp + off));
                if constexpr (PLANES == 2) l[u] = __ldcs(reinterpret_cast<const uint4*>(lp + off));
            }
        }
#pragma unroll
        for (int u = 0; u < D; ++u) nid[u] = q + D + u < len ? __ldg(ids + q + D + u) : 0u;
#pragma unroll
        for (int u = 0; u < D; ++u) {
            if (q + u < len) {
                const float sg = (id[u] & kCsNeg) ? -1.0f : 1.0f;
                const float2 sg2 = make_float2(sg, sg);
                uint16_t* stage = nullptr;
                if constexpr (STAGE) stage = a.plane + (size_t)(id[u] & ~kCsNeg) * a.ld_plane + c * VEC;
                float2 v[HV];
                cs_chunk_values<E, STAGE>(h[u], l[PLANES == 2 ? u : 0], stage, v);
#pragma unroll
                for (int e = 0; e < HV; ++e) {
                    acc[e] = __ffma2_rn(v[e], sg2, acc[e]);
                    csq[e] = __ffma2_rn(v[e], v[e], csq[e]);
                }
            }
        }
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        const int64_t j = c * VEC + e;
        if (j >= a.n) continue;
        a.SA[(size_t)j * a.ld_sa + b] = (double)((e & 1) ? acc[e / 2].y : acc[e / 2].x);
        a.col_part[(size_t)b * a.n + j] = (e & 1) ? csq[e / 2].y : csq[e / 2].x;
    }
}

// Rows at any alignment: as cs_rows_kernel, a thread owning kCsCols columns
// blockDim.x apart and reading them one element at a time (coalesced).  A
// batch's words are loaded before the first is decoded, which would wait for
// each: 50000 x 1001 FP16 into 1064 buckets 159 us decoded at the load.
constexpr int kCsCols = 4;

template <Elem E>
__global__ void __launch_bounds__(kCsThreads) cs_rows_any_kernel(CsRowsArgs a) {
    constexpr int D = CsElem<E>::PLANES == 2 ? kCsDepth / 2 : kCsDepth;
    const int64_t b = blockIdx.x;
    const int64_t j0 = (int64_t)blockIdx.y * blockDim.x * kCsCols + threadIdx.x;
    if (j0 >= a.n) return;
    const int32_t o0 = a.offsets[b], len = a.offsets[b + 1] - o0;
    const uint32_t* ids = a.perm + o0;
    float acc[kCsCols], csq[kCsCols];
#pragma unroll
    for (int k = 0; k < kCsCols; ++k) acc[k] = csq[k] = 0.0f;
    uint32_t nid[D];
#pragma unroll
    for (int u = 0; u < D; ++u) nid[u] = u < len ? __ldg(ids + u) : 0u;
    for (int32_t q = 0; q < len; q += D) {
        constexpr bool TWO = CsElem<E>::PLANES == 2;
        uint32_t id[D], h[D][kCsCols], l[TWO ? D : 1][kCsCols];
#pragma unroll
        for (int u = 0; u < D; ++u) {
            id[u] = nid[u];
            const size_t base = (size_t)(id[u] & ~kCsNeg) * a.ld;
#pragma unroll
            for (int k = 0; k < kCsCols; ++k) {
                const int64_t j = j0 + (int64_t)k * blockDim.x;
                // an element that is not summed or stored: the first of A
                const size_t at = q + u < len && j < a.n ? base + j : 0;
                if constexpr (E == Elem::F32) h[u][k] = __ldg(static_cast<const uint32_t*>(a.hi) + at);
                else h[u][k] = __ldg(static_cast<const uint16_t*>(a.hi) + at);
                if constexpr (TWO) l[u][k] = __ldg(static_cast<const uint16_t*>(a.lo) + at);
            }
        }
#pragma unroll
        for (int u = 0; u < D; ++u) nid[u] = q + D + u < len ? __ldg(ids + q + D + u) : 0u;
#pragma unroll
        for (int u = 0; u < D; ++u) {
            if (q + u < len) {
                const float sg = (id[u] & kCsNeg) ? -1.0f : 1.0f;
#pragma unroll
                for (int k = 0; k < kCsCols; ++k) {
                    const float v = word_value<E>(h[u][k], TWO ? l[TWO ? u : 0][k] : 0u);
                    acc[k] = fmaf(sg, v, acc[k]);
                    csq[k] = fmaf(v, v, csq[k]);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kCsCols; ++k) {
        const int64_t j = j0 + (int64_t)k * blockDim.x;
        if (j >= a.n) continue;
        a.SA[(size_t)j * a.ld_sa + b] = (double)acc[k];
        a.col_part[(size_t)b * a.n + j] = csq[k];
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Rows of at most kCsNarrowChunks chunks, of which there are few buckets
// (s ~ 4 n) of many rows: a thread per chunk would leave the memory system
// with a few KB in flight.  A CTA takes a whole bucket: all threads copy
// batches of kCsNarrowRows rows into a three-stage ring, and thread j then
// adds column j of the batch, row by row in order.  VECR: rows 16-byte
// aligned, copied in chunks; otherwise element by element.  1e6 x 64 bf16
// (256 buckets of ~3900 rows): 102 us, against 2.05 ms for a warp a bucket.
constexpr int kCsNarrowChunks = 32;
constexpr int kCsNarrowRows = 128;
constexpr int kCsNarrowBytes = 16 * 1024;  // a stage at most
constexpr int kCsNarrowStages = 3;

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

template <Elem E, bool STAGE, bool VECR>
__global__ void __launch_bounds__(256) cs_rows_narrow_kernel(CsRowsArgs a, int rows) {
    static_assert(!STAGE || (E == Elem::H16 && VECR), "staging writes FP32_16 wh planes");
    constexpr int VEC = CsElem<E>::VEC, ESZ = CsElem<E>::ESZ, PLANES = CsElem<E>::PLANES;
    constexpr int UNIT = VECR ? 16 : ESZ;  // bytes a copy moves
    extern __shared__ __align__(16) uint8_t ring[];
    __shared__ uint32_t sid[kCsNarrowStages][kCsNarrowRows];
    const int t = threadIdx.x, T = blockDim.x;
    const int nch = VECR ? (int)((a.n + VEC - 1) / VEC) : (int)a.n;  // copies a row and plane
    const int rb = nch * UNIT;                     // bytes of a row and plane in the ring
    const int plane_bytes = rows * rb;
    const int64_t b = blockIdx.x;
    const int32_t o0 = a.offsets[b], len = a.offsets[b + 1] - o0;
    const int nbat = (len + rows - 1) / rows;
    const size_t pitch = (size_t)a.ld * ESZ;
    auto issue = [&](int q) {
        if (q < nbat) {
            uint8_t* st = ring + (size_t)(q % kCsNarrowStages) * plane_bytes * PLANES;
            const int nr = len - q * rows < rows ? len - q * rows : rows;
#pragma unroll 8
            for (int e = t; e < nr * nch; e += T) {
                const int u = e / nch, c = e - u * nch;
                const uint32_t id = __ldg(a.perm + o0 + q * rows + u);
                const size_t off = (size_t)(id & ~kCsNeg) * pitch + (size_t)c * UNIT;
                const uint8_t* src = static_cast<const uint8_t*>(a.hi) + off;
                const uint8_t* srl = static_cast<const uint8_t*>(a.lo) + off;
                uint8_t* dst = st + u * rb + c * UNIT;
                if constexpr (VECR) {
                    cp_async16(dst, src);
                    if constexpr (PLANES == 2) cp_async16(dst + plane_bytes, srl);
                } else if constexpr (UNIT == 4) {
                    cp_async4(dst, src);
                } else {
                    *reinterpret_cast<uint16_t*>(dst) = __ldg(reinterpret_cast<const uint16_t*>(src));
                    if constexpr (PLANES == 2)
                        *reinterpret_cast<uint16_t*>(dst + plane_bytes) = __ldg(reinterpret_cast<const uint16_t*>(srl));
                }
                if (c == 0) sid[q % kCsNarrowStages][u] = id;
            }
        }
        cp_async_commit();
    };
    float acc = 0.0f, csq = 0.0f;
#pragma unroll
    for (int q = 0; q < kCsNarrowStages - 1; ++q) issue(q);
    for (int q = 0; q < nbat; ++q) {
        cp_async_wait<kCsNarrowStages - 2>();
        __syncthreads();  // batch q landed; the stage of batch q - 1 is free
        issue(q + kCsNarrowStages - 1);
        const int sl = q % kCsNarrowStages;
        uint8_t* st = ring + (size_t)sl * plane_bytes * PLANES;
        const int nr = len - q * rows < rows ? len - q * rows : rows;
        if constexpr (E == Elem::H16 && VECR) {
            // the fixed fp16 words in place (and to the plane)
            for (int e = t; e < nr * nch; e += T) {
                const int u = e / nch, c = e - u * nch;
                uint4* w = reinterpret_cast<uint4*>(st + u * rb + c * 16);
                uint4 h = *w;
                fix_half_chunk(h);
                *w = h;
                if constexpr (STAGE)
                    *reinterpret_cast<uint4*>(a.plane + (size_t)(sid[sl][u] & ~kCsNeg) * a.ld_plane + c * VEC) = h;
            }
            __syncthreads();
        }
        if (t < a.n) {
            constexpr Elem V = E == Elem::H16 && VECR ? Elem::F16 : E;  // what the ring holds
#pragma unroll 8
            for (int u = 0; u < nr; ++u) {
                const float sg = (sid[sl][u] & kCsNeg) ? -1.0f : 1.0f;
                const uint8_t* hw = st + u * rb + t * ESZ;
                float v;
                if constexpr (V == Elem::F32) v = *reinterpret_cast<const float*>(hw);
                else if constexpr (V == Elem::F16) v = half_bits_to_float(*reinterpret_cast<const uint16_t*>(hw));
                else if constexpr (V == Elem::H16) v = half_bits_to_float(half_only_bits(*reinterpret_cast<const uint16_t*>(hw)));
                else if constexpr (V == Elem::B16) v = u2f((uint32_t)*reinterpret_cast<const uint16_t*>(hw) << 16);
                else {
                    const uint32_t wh = *reinterpret_cast<const uint16_t*>(hw);
                    const uint32_t wr = *reinterpret_cast<const uint16_t*>(hw + plane_bytes);
                    v = V == Elem::A16 ? decode_fp32_16_exact_nb(wh, wr)
                                       : decode_fp32_bf16_exact(wh, wr, V == Elem::AB16R);
                }
                acc = fmaf(sg, v, acc);
                csq = fmaf(v, v, csq);
            }
        }
    }
    cp_async_wait<0>();
    if (t < a.n) {
        a.SA[(size_t)t * a.ld_sa + b] = (double)acc;
        a.col_part[(size_t)b * a.n + t] = csq;
    }
}

// Column sums of squares from the per-bucket FP32 partials: chunk q of the
// buckets sums its rows in bucket order into part[q][j] (FP64), then
// cs_colsq_final_kernel sums the chunks in order.
__global__ void cs_colsq_chunk_kernel(const float* __restrict__ col_part, int64_t s, int64_t n,
                                      int64_t per_chunk, double* __restrict__ part) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t q = blockIdx.y;
    if (j >= n) return;
    const int64_t b0 = q * per_chunk;
    const int64_t b1 = (b0 + per_chunk) < s ? (b0 + per_chunk) : s;
    double t = 0.0;
    for (int64_t b = b0; b < b1; ++b) t += (double)col_part[(size_t)b * n + j];
    part[(size_t)q * n + j] = t;
}

__global__ void cs_colsq_final_kernel(const double* __restrict__ part, int64_t chunks, int64_t n,
                                      double* __restrict__ colsq) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double t = 0.0;
    for (int64_t q = 0; q < chunks; ++q) t += part[(size_t)q * n + j];
    colsq[j] = t;
}

// Column-major owner sums: block per column, warps over buckets, lanes
// over the bucket's rows (gathered down the contiguous column).
template <Elem E>
__global__ void __launch_bounds__(256) cs_cols_kernel(const void* hi, const void* lo, int64_t n,
                                                      int64_t ld, int64_t s,
                                                      const int32_t* __restrict__ offsets,
                                                      const uint32_t* __restrict__ perm,
                                                      double* __restrict__ SA, int64_t ld_sa,
                                                      double* __restrict__ fro_part,
                                                      double* __restrict__ colsq) {
    __shared__ double smf[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t j = blockIdx.x;
    const size_t cbase = (size_t)j * ld;
    double f2 = 0.0;
    for (int64_t b = w; b < s; b += 8) {
        const int32_t o0 = offsets[b], o1 = offsets[b + 1];
        double acc = 0.0;
        int32_t q = o0 + lane;
        if (o1 - o0 > 32) {  // four of a long bucket's rows in flight
            for (; q + 96 < o1; q += 128) {
                uint32_t r[4];
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) r[u] = perm[q + 32 * u];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = load_elem<E>(hi, lo, cbase + (r[u] & ~kCsNeg));
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double a = (double)u2f(__float_as_uint(v[u]) ^ (r[u] & kCsNeg));
                    acc += a;
                    f2 += a * a;
                }
            }
        }
#pragma unroll 1
        for (; q < o1; q += 32) {
            const uint32_t r = perm[q];
            float v[1];
            load_elems<E, 1>(hi, lo, cbase + (r & ~kCsNeg), 0, v);
            const double a = (double)u2f(__float_as_uint(v[0]) ^ (r & kCsNeg));  // the row's sign on the value
            acc += a;
            f2 += a * a;
        }
        acc = warp_sum(acc);
        if (lane == 0) SA[(size_t)j * ld_sa + b] = acc;
    }
    f2 = warp_sum(f2);
    if (lane == 0) smf[w] = f2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += smf[k];
        fro_part[blockIdx.x] = t;
        if (colsq) colsq[blockIdx.x] = t;
    }
}

__global__ void cs_fro_reduce_kernel(const double* __restrict__ part, int64_t np,
                                     double* __restrict__ out) {
    __shared__ double sm[32];
    double s = 0.0;
    for (int64_t k = threadIdx.x; k < np; k += blockDim.x) s += part[k];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        t = warp_sum(t);
        if (threadIdx.x == 0) *out = t;
    }
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

CsScratch cs_layout(void* base, int64_t m, int64_t s, int64_t fro_parts, int64_t col_parts) {
    CsScratch c;
    size_t off = 0;
    char* p = static_cast<char*>(base);
    auto take = [&](size_t bytes) {
        char* q = p ? p + off : nullptr;
        off += align256(bytes);
        return q;
    };
    c.bucket = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (m > 0 ? m : 1)));
    c.sign = reinterpret_cast<int8_t*>(take(m > 0 ? m : 1));
    c.cnt = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (size_t)cs_segments(m, s) * s));
    c.counts = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (s + 1)));
    c.offsets = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (s + 1)));
    c.cursor = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (s + 1)));
    c.perm = reinterpret_cast<uint32_t*>(take(sizeof(int32_t) * (m > 0 ? m : 1)));
    c.fro_part = reinterpret_cast<double*>(take(sizeof(double) * (fro_parts > 0 ? fro_parts : 1)));
    c.col_part = reinterpret_cast<double*>(take(sizeof(double) * (col_parts > 0 ? col_parts : 1)));
    c.bytes = off;
    return c;
}

int64_t cs_col_part_rows(int64_t m, int64_t s) {
    // row-major: s x n FP32 per-bucket partials, then n FP64 column sums, from
    // entry (s n + 1) / 2 <= n (s + 1) / 2 on
    const int64_t rows = (s + 1) / 2 + 1;
    int64_t csr = (int64_t)sm_count() * 2;             // CSR row-chunk blocks
    const int64_t cm = (m + 63) / 64;
    if (csr > cm) csr = cm;
    return rows > csr ? rows : csr;
}

// Upper bound of the owner-sum partial count over both layouts and the
// CSR path, so one size query serves all callers.
int64_t cs_fro_parts(int64_t m, int64_t s) {
    (void)m;
    const int64_t rows = ((s + 7) / 8) * 64;  // row-major: blocks x panels (n <= 64 panels cap)
    const int64_t csr = (s + 7) / 8;
    int64_t v = rows > csr ? rows : csr;
    return v < 65536 ? 65536 : v;  // column-major: one per column (n <= 65536)
}

static bool cs_grid(int64_t m, int* g) {
    int64_t b = (m + 255) / 256;
    int64_t cap = (int64_t)sm_count() * 8;
    if (b > cap) b = cap;
    *g = (int)(b < 1 ? 1 : b);
    return true;
}

// Row segments of the counting sort: enough single-warp placements to fill
// the GPU (eight a SM), at least 256 rows each, and a count matrix (segments
// x s) of at most 4 M words, which stays in L2.  0: s exceeds the shared
// counters of a CTA.
int64_t cs_segments(int64_t m, int64_t s) {
    if (s > kCsMaxCounted || m <= 0) return 0;
    int64_t g = (int64_t)sm_count() * 8;
    if (g > (m + 255) / 256) g = (m + 255) / 256;
    if (g > ((int64_t)4 << 20) / s) g = ((int64_t)4 << 20) / s;
    return g < 1 ? 1 : g;
}

// Steps 1-3 (shared by the dense and CSR owner sums): offsets and perm.
// The stable counting sort replaces a global histogram, an unordered scatter
// and a sort of each bucket, whose cost grows with the square of a bucket's
// length past kCsSortCap rows: 58 ms of it at 1e6 rows in 256 buckets, now
// 32 us for all three kernels; 116 us -> 40 us at 1e6 rows in 4000 buckets.
tomos_status cs_bucketize(int64_t m, int64_t s, uint64_t bseed, uint64_t sseed, const CsScratch& c,
                          cudaStream_t st, int64_t row0) {
    const int64_t nseg = cs_segments(m, s);
    if (nseg > 0) {
        const int64_t per = (m + nseg - 1) / nseg;
        const size_t smem = sizeof(int32_t) * (size_t)s;
        if (smem > 48 * 1024) {
            TOMOS_CUDA_TRY(cudaFuncSetAttribute(cs_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            TOMOS_CUDA_TRY(cudaFuncSetAttribute(cs_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        }
        cs_count_kernel<<<(unsigned)nseg, 256, smem, st>>>(m, per, (int32_t)s, bseed, sseed, row0,
                                                           reinterpret_cast<uint32_t*>(c.bucket), c.cnt);
        TOMOS_LAUNCH_CHECK("cs_count_kernel");
        cs_segment_scan_kernel<<<(unsigned)((s + 31) / 32), 1024, 0, st>>>(c.cnt, (int)nseg, (int32_t)s, c.counts);
        TOMOS_LAUNCH_CHECK("cs_segment_scan_kernel");
        cs_scan_kernel<<<1, 1024, 0, st>>>(c.counts, s, c.offsets);
        TOMOS_LAUNCH_CHECK("cs_scan_kernel");
        cs_place_kernel<<<(unsigned)nseg, 256, smem, st>>>(m, per, (int32_t)s,
                                                           reinterpret_cast<const uint32_t*>(c.bucket), c.cnt,
                                                           c.offsets, c.perm);
        TOMOS_LAUNCH_CHECK("cs_place_kernel");
        return TOMOS_OK;
    }
    int g;
    cs_grid(m, &g);
    TOMOS_CUDA_TRY(cudaMemsetAsync(c.counts, 0, sizeof(int32_t) * (s + 1), st));
    TOMOS_CUDA_TRY(cudaMemsetAsync(c.cursor, 0, sizeof(int32_t) * (s + 1), st));
    cs_hash_kernel<<<g, 256, 0, st>>>(m, s, bseed, sseed, row0, c.bucket, c.sign, c.counts);
    TOMOS_LAUNCH_CHECK("cs_hash_kernel");
    cs_scan_kernel<<<1, 1024, 0, st>>>(c.counts, s, c.offsets);
    TOMOS_LAUNCH_CHECK("cs_scan_kernel");
    cs_scatter_kernel<<<g, 256, 0, st>>>(m, c.bucket, c.sign, c.offsets, c.cursor, c.perm);
    TOMOS_LAUNCH_CHECK("cs_scatter_kernel");
    cs_sort_kernel<<<(unsigned)((s + kCsSortWarps - 1) / kCsSortWarps), kCsSortWarps * 32, 0, st>>>(
        s, c.offsets, c.perm);
    TOMOS_LAUNCH_CHECK("cs_sort_kernel");
    return TOMOS_OK;
}

// Whether the staged owner sums can read A (16-byte aligned rows).
static bool rows_vec_ok(const tomos_dense* A, const void* lo, int esz) {
    bool vec = ((A->ld * esz) % 16 == 0) && (reinterpret_cast<uintptr_t>(A->values) % 16 == 0);
    if (vec && lo) vec = reinterpret_cast<uintptr_t>(lo) % 16 == 0;
    return vec;
}

// The row-major owner sums and the reductions behind them: SA, colsq and
// fro2 (both optional).
template <Elem E, bool STAGE>
static tomos_status launch_rows(const tomos_dense* A, const void* lo, int64_t s, const CsScratch& c,
                                double* SA, int64_t ld_sa, double* colsq, double* fro2,
                                uint16_t* plane, int64_t ld_plane, cudaStream_t st) {
    constexpr int VEC = CsElem<E>::VEC, PLANES = CsElem<E>::PLANES;
    const int64_t n = A->cols;
    CsRowsArgs a;
    a.hi = A->values;
    a.lo = lo;
    a.n = n;
    a.ld = A->ld;
    a.s = s;
    a.offsets = c.offsets;
    a.perm = c.perm;
    a.SA = SA;
    a.ld_sa = ld_sa;
    a.col_part = reinterpret_cast<float*>(c.col_part);
    a.plane = plane;
    a.ld_plane = ld_plane;
    const int64_t nch = (n + VEC - 1) / VEC;
    const bool vec = rows_vec_ok(A, lo, CsElem<E>::ESZ);
    if (nch <= kCsNarrowChunks) {
        const int rb = (int)(vec ? nch * 16 : n * CsElem<E>::ESZ);
        int rows = kCsNarrowBytes / (rb * PLANES);
        if (rows > kCsNarrowRows) rows = kCsNarrowRows;
        const size_t smem = (size_t)kCsNarrowStages * rows * rb * PLANES;
        void (*kern)(CsRowsArgs, int) = cs_rows_narrow_kernel<E, STAGE, true>;
        if constexpr (!STAGE)
            if (!vec) kern = cs_rows_narrow_kernel<E, false, false>;
        TOMOS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<(unsigned)s, n <= 128 ? 128 : 256, smem, st>>>(a, rows);
        TOMOS_LAUNCH_CHECK("cs_rows_narrow_kernel");
    } else {
        // threads: the chunks (or columns / kCsCols) of a row in whole
        // warps, split over CTAs of at most kCsThreads
        const int64_t units = vec ? nch : (n + kCsCols - 1) / kCsCols;
        const int64_t panels = (units + kCsThreads - 1) / kCsThreads;
        const int64_t threads = ((units + panels - 1) / panels + 31) / 32 * 32;
        const dim3 grid((unsigned)s, (unsigned)panels);
        if (vec)
            cs_rows_kernel<E, STAGE><<<grid, (unsigned)threads, 0, st>>>(a);
        else
            cs_rows_any_kernel<E><<<grid, (unsigned)threads, 0, st>>>(a);
        TOMOS_LAUNCH_CHECK("cs_rows_kernel");
    }
    // colsq (into the caller's buffer, or the scratch after the s n FP32
    // partials: an odd count is rounded up, doubles start on 8 bytes), then
    // fro2 as their sum
    double* cs = colsq ? colsq : c.col_part + (s * n + 1) / 2;
    int64_t chunks = (s + 63) / 64;
    const int64_t cap = cs_fro_parts(A->rows, s) / (n > 0 ? n : 1);
    if (chunks > cap) chunks = cap > 0 ? cap : 1;
    const int64_t per = (s + chunks - 1) / chunks;
    chunks = (s + per - 1) / per;
    cs_colsq_chunk_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)chunks), 256, 0, st>>>(
        a.col_part, s, n, per, c.fro_part);
    TOMOS_LAUNCH_CHECK("cs_colsq_chunk_kernel");
    cs_colsq_final_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(c.fro_part, chunks, n, cs);
    TOMOS_LAUNCH_CHECK("cs_colsq_final_kernel");
    if (fro2) {
        cs_fro_reduce_kernel<<<1, 256, 0, st>>>(cs, n, fro2);
        TOMOS_LAUNCH_CHECK("cs_fro_reduce_kernel");
    }
    return TOMOS_OK;
}

template <Elem E>
static void launch_cols(const tomos_dense* A, const void* lo, int64_t s, const CsScratch& c,
                        double* SA, int64_t ld_sa, double* colsq, cudaStream_t st) {
    cs_cols_kernel<E><<<(unsigned)A->cols, 256, 0, st>>>(A->values, lo, A->cols, A->ld, s, c.offsets,
                                                         c.perm, SA, ld_sa, c.fro_part, colsq);
}

}  // namespace tomos_b200

using namespace tomos_b200;

extern "C" {

tomos_status tomos_countsketch_hash(int64_t m, int64_t s, uint64_t bucket_seed, uint64_t sign_seed,
                                    int32_t* bucket, int8_t* sign, void* stream) {
    if (m < 0 || s <= 0) return fail(TOMOS_ERR_INVALID, "countsketch_hash: need m >= 0, s > 0");
    if (m == 0) return TOMOS_OK;
    if (m > 0x7fffffffLL) return fail(TOMOS_ERR_INVALID, "countsketch_hash: m exceeds int32");
    if (!bucket || !sign) return fail(TOMOS_ERR_INVALID, "countsketch_hash: null output");
    int g;
    cs_grid(m, &g);
    cs_hash_kernel<<<g, 256, 0, as_stream(stream)>>>(m, s, bucket_seed, sign_seed, 0, bucket, sign,
                                                     nullptr);
    TOMOS_LAUNCH_CHECK("cs_hash_kernel");
    return TOMOS_OK;
}

size_t tomos_countsketch_scratch_bytes(int64_t m, int64_t cols, int64_t s) {
    if (m < 0 || s <= 0 || cols < 0) return 0;
    return cs_layout(nullptr, m, s, cs_fro_parts(m, s), cs_col_part_rows(m, s) * cols).bytes;
}

}  // extern "C"

namespace tomos_b200 {

// tomos_countsketch_apply, and with `plane` the staged fp16 copy of an
// FP32_16 wh plane written by the same pass (tomos_countsketch_apply_stage).
static tomos_status countsketch_apply(const tomos_dense* A, int32_t tier, int64_t s,
                                      uint64_t bucket_seed, uint64_t sign_seed, double* SA,
                                      int64_t ld_sa, double* fro2, double* colsq, void* scratch,
                                      size_t scratch_bytes, void* stream, uint16_t* plane,
                                      int64_t ld_plane, int64_t row0 = 0) {
    if (!A || s <= 0) return fail(TOMOS_ERR_INVALID, "countsketch_apply: need A and s > 0");
    if (A->layout != TOMOS_ROW_MAJOR && A->layout != TOMOS_COL_MAJOR)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply: bad layout");
    const int64_t m = A->rows, n = A->cols;
    if (m < 0 || n < 0) return fail(TOMOS_ERR_INVALID, "countsketch_apply: negative size");
    if (m > 0x7fffffffLL) return fail(TOMOS_ERR_INVALID, "countsketch_apply: m exceeds int32");
    if (ld_sa < s) return fail(TOMOS_ERR_INVALID, "countsketch_apply: ld_sa < s");
    const int64_t inner = A->layout == TOMOS_ROW_MAJOR ? n : m;
    if (A->ld < inner) return fail(TOMOS_ERR_INVALID, "countsketch_apply: bad leading dimension");
    if (A->layout == TOMOS_COL_MAJOR && n > 65536)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply: column-major n > 65536");
    if (A->layout == TOMOS_ROW_MAJOR && n > 64 * 256)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply: row-major n > 16384");
    Elem e;
    std::string why;
    if (!resolve_elem(A, tier, &e, &why)) return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply: " + why);
    cudaStream_t st = as_stream(stream);
    if (n == 0) return TOMOS_OK;
    if (!SA) return fail(TOMOS_ERR_INVALID, "countsketch_apply: null SA");
    if (m == 0) {
        for (int64_t j = 0; j < n; ++j)
            TOMOS_CUDA_TRY(cudaMemsetAsync(SA + j * ld_sa, 0, sizeof(double) * s, st));
        if (fro2) TOMOS_CUDA_TRY(cudaMemsetAsync(fro2, 0, sizeof(double), st));
        if (colsq) TOMOS_CUDA_TRY(cudaMemsetAsync(colsq, 0, sizeof(double) * n, st));
        return TOMOS_OK;
    }
    const int64_t col_parts = cs_col_part_rows(m, s) * n;
    CsScratch need = cs_layout(nullptr, m, s, cs_fro_parts(m, s), col_parts);
    if (!scratch || scratch_bytes < need.bytes)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply: scratch too small (need " +
                                           std::to_string(need.bytes) + " bytes)");
    CsScratch c = cs_layout(scratch, m, s, cs_fro_parts(m, s), col_parts);
    tomos_status rc = cs_bucketize(m, s, bucket_seed, sign_seed, c, st, row0);
    if (rc) return rc;
    const void* lo = (e == Elem::A16 || e == Elem::AB16 || e == Elem::AB16R) ? dense_lo_plane(A)
                                                                             : nullptr;
    int64_t nparts;
    if (plane && !rows_vec_ok(A, lo, 2))
        return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply_stage: rows of A not 16-byte aligned");
    if (A->layout == TOMOS_ROW_MAJOR) {
        // colsq and fro2 come with the owner sums
#define TOMOS_CS_ROWS(EE) launch_rows<EE, false>(A, lo, s, c, SA, ld_sa, colsq, fro2, nullptr, 0, st)
        switch (e) {
            case Elem::F32: return TOMOS_CS_ROWS(Elem::F32);
            case Elem::H16:
                return plane ? launch_rows<Elem::H16, true>(A, lo, s, c, SA, ld_sa, colsq, fro2, plane, ld_plane, st)
                             : TOMOS_CS_ROWS(Elem::H16);
            case Elem::A16: return TOMOS_CS_ROWS(Elem::A16);
            case Elem::F16: return TOMOS_CS_ROWS(Elem::F16);
            case Elem::B16: return TOMOS_CS_ROWS(Elem::B16);
            case Elem::AB16: return TOMOS_CS_ROWS(Elem::AB16);
            case Elem::AB16R: return TOMOS_CS_ROWS(Elem::AB16R);
            default: return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply: element type");
        }
#undef TOMOS_CS_ROWS
    } else {
        switch (e) {
            case Elem::F32: launch_cols<Elem::F32>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::H16: launch_cols<Elem::H16>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::A16: launch_cols<Elem::A16>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::F16: launch_cols<Elem::F16>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::B16: launch_cols<Elem::B16>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::AB16: launch_cols<Elem::AB16>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            case Elem::AB16R: launch_cols<Elem::AB16R>(A, lo, s, c, SA, ld_sa, colsq, st); break;
            default: return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply: element type");
        }
        nparts = n;
    }
    TOMOS_LAUNCH_CHECK("countsketch owner sums");
    if (fro2) {
        cs_fro_reduce_kernel<<<1, 256, 0, st>>>(c.fro_part, nparts, fro2);
        TOMOS_LAUNCH_CHECK("cs_fro_reduce_kernel");
    }
    return TOMOS_OK;
}

}  // namespace tomos_b200

extern "C" {

tomos_status tomos_countsketch_apply(const tomos_dense* A, int32_t tier, int64_t s,
                                     uint64_t bucket_seed, uint64_t sign_seed, double* SA,
                                     int64_t ld_sa, double* fro2, double* colsq, void* scratch,
                                     size_t scratch_bytes, void* stream) {
    return countsketch_apply(A, tier, s, bucket_seed, sign_seed, SA, ld_sa, fro2, colsq, scratch,
                             scratch_bytes, stream, nullptr, 0);
}

tomos_status tomos_countsketch_apply_shard(const tomos_dense* A, int32_t tier, int64_t s,
                                           uint64_t bucket_seed, uint64_t sign_seed, int64_t row0,
                                           double* SA, int64_t ld_sa, double* fro2, double* colsq,
                                           void* plane, int64_t ld_plane, void* scratch,
                                           size_t scratch_bytes, void* stream) {
    if (row0 < 0) return fail(TOMOS_ERR_INVALID, "countsketch_apply_shard: negative row0");
    if (plane) {
        if (!A || A->numeric != TOMOS_FP32_16 || A->layout != TOMOS_ROW_MAJOR || tier != TOMOS_TIER_HALF)
            return fail(TOMOS_ERR_INVALID,
                        "countsketch_apply_shard: a staged plane needs a row-major FP32_16 A at the HALF tier");
        if (reinterpret_cast<uintptr_t>(plane) % 16 != 0 || ld_plane < A->cols || ld_plane % 8 != 0)
            return fail(TOMOS_ERR_INVALID,
                        "countsketch_apply_shard: plane must be 16-byte aligned with ld_plane a multiple of 8 "
                        "and >= cols");
        if (!rows_vec_ok(A, nullptr, 2))
            return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply_shard: rows of A not 16-byte aligned");
    }
    return countsketch_apply(A, tier, s, bucket_seed, sign_seed, SA, ld_sa, fro2, colsq, scratch,
                             scratch_bytes, stream, static_cast<uint16_t*>(plane), ld_plane, row0);
}

tomos_status tomos_countsketch_apply_stage(const tomos_dense* A, int64_t s, uint64_t bucket_seed,
                                           uint64_t sign_seed, double* SA, int64_t ld_sa,
                                           double* fro2, double* colsq, void* plane,
                                           int64_t ld_plane, void* scratch, size_t scratch_bytes,
                                           void* stream) {
    if (!A || A->numeric != TOMOS_FP32_16 || A->layout != TOMOS_ROW_MAJOR)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply_stage: A must be row-major FP32_16");
    if (!plane || reinterpret_cast<uintptr_t>(plane) % 16 != 0)
        return fail(TOMOS_ERR_INVALID, "countsketch_apply_stage: plane must be 16-byte aligned");
    if (ld_plane < A->cols || ld_plane % 8 != 0)
        return fail(TOMOS_ERR_INVALID,
                    "countsketch_apply_stage: ld_plane must be a multiple of 8 and >= cols");
    if (!rows_vec_ok(A, nullptr, 2))
        return fail(TOMOS_ERR_UNSUPPORTED, "countsketch_apply_stage: rows of A not 16-byte aligned");
    return countsketch_apply(A, TOMOS_TIER_HALF, s, bucket_seed, sign_seed, SA, ld_sa, fro2, colsq,
                             scratch, scratch_bytes, stream, static_cast<uint16_t*>(plane), ld_plane);
}

}  // extern "C"
