// qr_gemm.cuh -- FP64 products of the blocked QR on the tensor cores
// (mma.sync m16n8k8 f64), and the pieces that turn a block of panels into
// one compact-WY transform.
//
// A block of kQrBlock columns is factored panel by panel (32 columns, the
// trailing update restricted to the block); its reflectors V (k_rem x 256)
// and the panels' 32 x 32 factors T_p then make the block's
// H_1 ... H_256 = I - V T V^T, with T upper triangular and
//   T = [[T_<j, -T_<j (V_<j^T V_j) T_j], [0, T_j]]    (j = 1 .. 7),
// and the columns right of the block get C <- (I - V T^T V^T) C as three
// products: Z = V T, W = Z^T C, C -= V W.  Each reads C once per block
// instead of twice per panel.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "mbarrier.cuh"  // smem_addr

namespace tomos_b200 {

constexpr int kQrBlock = 256;     // columns per block of the blocked QR
constexpr int kGbm = 128;         // GEMM CTA tile rows
constexpr int kGbn = 64;          // GEMM CTA tile columns
constexpr int kGbk = 16;          // k per stage
constexpr int kGpad = 4;          // row padding (doubles) of the stage tiles
constexpr int kGstages = 3;
constexpr int kGmaxSplits = 16;
constexpr int kGa = kGbm * (kGbk + kGpad) > kGbk * (kGbm + kGpad) ? kGbm * (kGbk + kGpad)
                                                                 : kGbk * (kGbm + kGpad);
constexpr int kGb = kGbn * (kGbk + kGpad);
constexpr int kGstage = kGa + kGb;
constexpr size_t kGemmSmem = sizeof(double) * kGstage * kGstages;

__device__ __forceinline__ void g_cp_async8(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void g_cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
// Two neighbouring values of which the first n (0, 1, 2) exist, the others
// zero; vec: both addresses are 16-byte aligned.
__device__ __forceinline__ void g_copy_pair(double* dst, const double* src, const double* safe, int n, bool vec) {
    if (vec && n == 2) {
        g_cp_async16(dst, src);
    } else {
        g_cp_async8(dst, n > 0 ? src : safe, n > 0);
        g_cp_async8(dst + 1, n > 1 ? src + 1 : safe, n > 1);
    }
}
__device__ __forceinline__ void g_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void g_cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// D += A B for one m16n8k8 FP64 tile: with g = lane / 4, q = lane % 4,
// a = A[g][q], A[g + 8][q], A[g][q + 4], A[g + 8][q + 4]; b = B[q][g],
// B[q + 4][g]; d = D[g][2q], D[g][2q + 1], D[g + 8][2q], D[g + 8][2q + 1].
__device__ __forceinline__ void g_dmma1688(double* d, const double* a, const double* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// D (M x N, column-major, ld ldd) = alpha * op(A) B + beta * D, B
// column-major K x N.  KMAJOR: op(A) = A^T with A column-major K x M;
// otherwise A is column-major M x K.  CTA tile 128 x 64, k-steps of 16
// through kGstages shared-memory stages filled by asynchronous copies of
// pairs (16 bytes where the operand is aligned, zero-filled past the edges),
// one barrier a stage (12000 x 3000 symmetric product and its updates 3.9 ms;
// 4.5 ms with 8-byte copies and two barriers); 8 warps, each 32 x 32 = two by
// four m16n8k8 tiles.  Split-K: CTA z sums k in [z kc, (z + 1) kc); with
// gridDim.z > 1 it writes its partial to P + z M N (ld M) for
// qr_gemm_reduce_kernel.  sub: D -= op(A) B instead (alpha and beta
// unused): the accumulators start from the D tile, loaded while the first
// stages are in flight, and A enters negated.
struct GemmArgs {
    const double* A;
    int64_t lda;
    const double* B;
    int64_t ldb;
    double* D;
    int64_t ldd;
    double* P;
    int64_t M, N, K, kc;
    double alpha, beta;
    int sub;
    int upper;  // skip the tiles wholly below the diagonal (a symmetric product's other half)
};

template <bool KMAJOR>
__global__ void __launch_bounds__(256, 2) qr_gemm_kernel(GemmArgs g) {
    extern __shared__ __align__(16) double gsm[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int gq = lane >> 2, qq = lane & 3;
    const int wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
    const int64_t m0 = (int64_t)blockIdx.x * kGbm, n0 = (int64_t)blockIdx.y * kGbn;
    if (g.upper && m0 > n0 + kGbn - 1) return;
    const int64_t kb = (int64_t)blockIdx.z * g.kc;
    const int64_t ke = kb + g.kc < g.K ? kb + g.kc : g.K;
    const int nk = ke > kb ? (int)((ke - kb + kGbk - 1) / kGbk) : 0;
    const bool avec = g.lda % 2 == 0 && reinterpret_cast<uintptr_t>(g.A) % 16 == 0;
    const bool bvec = g.ldb % 2 == 0 && reinterpret_cast<uintptr_t>(g.B) % 16 == 0;
    auto left = [](int64_t at, int64_t end) { return at + 1 < end ? 2 : (at < end ? 1 : 0); };
    auto issue = [&](int s, int64_t k0) {
        double* As = gsm + s * kGstage;
        double* Bs = As + kGa;
#pragma unroll
        for (int i = 0; i < kGbm * kGbk / 512; ++i) {
            const int e = t + i * 256;
            if (KMAJOR) {  // pairs along K
                const int m = e >> 3, kk = (e & 7) * 2;
                const int64_t gm = m0 + m, gk = k0 + kk;
                g_copy_pair(As + m * (kGbk + kGpad) + kk, g.A + gk + gm * g.lda, g.A, gm < g.M ? left(gk, ke) : 0, avec);
            } else {       // pairs along M
                const int m = (e & (kGbm / 2 - 1)) * 2, kk = e >> 6;
                const int64_t gm = m0 + m, gk = k0 + kk;
                g_copy_pair(As + kk * (kGbm + kGpad) + m, g.A + gm + gk * g.lda, g.A, gk < ke ? left(gm, g.M) : 0, avec);
            }
        }
#pragma unroll
        for (int i = 0; i < kGbn * kGbk / 512; ++i) {
            const int e = t + i * 256, nn = e >> 3, kk = (e & 7) * 2;
            const int64_t gn = n0 + nn, gk = k0 + kk;
            g_copy_pair(Bs + nn * (kGbk + kGpad) + kk, g.B + gk + gn * g.ldb, g.B, gn < g.N ? left(gk, ke) : 0, bvec);
        }
        g_cp_async_commit();
    };
    double acc[2][4][4];
#pragma unroll
    for (int s = 0; s < kGstages - 1; ++s) {
        if (s < nk) issue(s, kb + (int64_t)s * kGbk);
        else g_cp_async_commit();
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int64_t row = m0 + wm + a * 16 + gq + 8 * (u >> 1);
                const int64_t col = n0 + wn + b * 8 + 2 * qq + (u & 1);
                acc[a][b][u] = (g.sub && row < g.M && col < g.N) ? g.D[row + col * g.ldd] : 0.0;
            }
    const double asg = g.sub ? -1.0 : 1.0;
    for (int i = 0; i < nk; ++i) {
        g_cp_async_wait<kGstages - 2>();
        __syncthreads();  // stage i landed, and stage i - 1 was read by all
        const int ni = i + kGstages - 1;
        if (ni < nk) issue(ni % kGstages, kb + (int64_t)ni * kGbk);
        else g_cp_async_commit();
        const double* As = gsm + (i % kGstages) * kGstage;
        const double* Bs = As + kGa;
#pragma unroll
        for (int ks = 0; ks < kGbk / 8; ++ks) {
            double a[2][4], b[4][2];
#pragma unroll
            for (int im = 0; im < 2; ++im)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int row = wm + im * 16 + gq + 8 * (u & 1), kk = ks * 8 + qq + 4 * (u >> 1);
                    a[im][u] = asg * (KMAJOR ? As[row * (kGbk + kGpad) + kk] : As[kk * (kGbm + kGpad) + row]);
                }
#pragma unroll
            for (int in = 0; in < 4; ++in)
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    b[in][u] = Bs[(wn + in * 8 + gq) * (kGbk + kGpad) + ks * 8 + qq + 4 * u];
#pragma unroll
            for (int im = 0; im < 2; ++im)
#pragma unroll
                for (int in = 0; in < 4; ++in) g_dmma1688(acc[im][in], a[im], b[in]);
        }
    }
    g_cp_async_wait<0>();
    const bool split = gridDim.z > 1;
#pragma unroll
    for (int im = 0; im < 2; ++im)
#pragma unroll
        for (int in = 0; in < 4; ++in)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int64_t row = m0 + wm + im * 16 + gq + 8 * (u >> 1);
                const int64_t col = n0 + wn + in * 8 + 2 * qq + (u & 1);
                if (row >= g.M || col >= g.N) continue;
                if (split) {
                    g.P[(size_t)blockIdx.z * g.M * g.N + row + col * g.M] = acc[im][in][u];
                } else if (g.sub) {
                    g.D[row + col * g.ldd] = acc[im][in][u];
                } else {
                    double v = g.alpha * acc[im][in][u];
                    if (g.beta != 0.0) v += g.beta * g.D[row + col * g.ldd];
                    g.D[row + col * g.ldd] = v;
                }
            }
}

// D = alpha * sum_z P[z] + beta * D, the splits summed in order.  D may be
// P[0] (ldd = M): a thread reads an entry's partials before it writes the entry.
__global__ void qr_gemm_reduce_kernel(const double* P, int splits, int64_t M, int64_t N,
                                      double alpha, double beta, double* D, int64_t ldd) {
    const int64_t total = M * N;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int z = 0; z < splits; ++z) s += P[(size_t)z * total + e];
        const int64_t row = e % M, col = e / M;
        double v = alpha * s;
        if (beta != 0.0) v += beta * D[row + col * ldd];
        D[row + col * ldd] = v;
    }
}

// Vb (krem x w, ld ldv) = the block's reflectors: V(i, a) = A[j0 + a][j0 + i]
// below the diagonal, 1 on it, 0 above.
__global__ void qr_copy_v_kernel(const double* __restrict__ A, int64_t ld, int64_t j0, int64_t krem, int w,
                                 double* __restrict__ Vb, int64_t ldv) {
    const int64_t total = krem * w;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e % krem, a = e / krem;
        Vb[i + a * ldv] = i > a ? A[(size_t)(j0 + a) * ld + j0 + i] : (i == a ? 1.0 : 0.0);
    }
}

// The block's T (w x w, column-major ld w) before its off-diagonal blocks:
// the panels' factors Tp[p] (32 x 32, T(a, b) at [b * 32 + a]) on the
// diagonal, zeros elsewhere.  T is the inverse of the block upper
// triangular L with diagonal blocks T_p^{-1} and off-diagonal blocks those
// of V^T V (the merge T_<j,j = -T_<j (V_<j^T V_j) T_j); the recursive
// inversion levels of the triangular inverse fill the rest.
__global__ void qr_block_t_init_kernel(const double* __restrict__ Tp, int w, double* __restrict__ T) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < w * w; e += gridDim.x * blockDim.x) {
        const int r = e % w, c = e / w;
        T[e] = r / 32 == c / 32 ? Tp[(size_t)(c / 32) * 1024 + (c % 32) * 32 + (r % 32)] : 0.0;
    }
}

}  // namespace tomos_b200
