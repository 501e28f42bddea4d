// dense_bottom.cuh -- the bottom of the V-cycle as one dense product.
//
// From a zero guess, the part of the cycle from level f down is linear in its
// right-hand side: x_f = B b_f with a fixed n_f x n_f matrix B.  Level by
// level it costs five small kernels a level (2 us of launch and drain each,
// 4 to 17 us for the coarsest solve or the cluster tail), whatever their
// size; one product with B takes 3.9 us (100^2; 192^3: 4.5) to 8.7
// us (1024^2), for 8 columns 27 us (96^3, smoothed aggregation).  Setup forms B
// once, in FP64 from the FP64 hierarchy, upwards from the inverse of the
// coarsest matrix:
//
//     T = R (I - A D)         restriction of the first sweep's residual
//     E = B_c T               the level below
//     X = D + P E             first sweep plus coarse correction
//     B = X + D (I - A X)     post-sweep
//
// with D the smoother's scaled inverse diagonal (no sweeps: B = P B_c R).
// B stays in FP64 under an FP32 cycle too, as the coarsest inverse does: on a
// nearly singular operator its entries are dominated by the large multiple of
// the near-null vector's projector, and rounded to FP32 they lose what the
// cycle does to everything else (graph Laplacian + 1e-7 on 40^3: error off
// the constant 2e-4, in FP64 8e-8).  On the same schedules an FP32 cycle
// takes as long with either (192^3 478.3 and 478.6 us, 1024^2 143.4 and 143.3),
// k = 8 columns of 96^3 1.5% longer (11.5 -> 11.7 ms a solve).
#pragma once

#include "rb_common.cuh"

namespace rb {

// Bytes of the largest B: 16 MB, of which the L2 (126 MB) keeps what a
// cycle's other levels leave; a product at that size reads about as long as
// two of the launches it replaces take.
constexpr size_t kDenseBytes = (size_t)16 << 20;

// Row length of B: rows start on 16-byte boundaries.
inline int dense_ld(int n) { return (n + 1) & ~1; }

// Row `row` of B b for one warp: 16 bytes a lane and step, rows padded with
// zeros to ld, b read only below n; every lane gets the sum.
template <typename T>
__device__ __forceinline__ double dense_row(int n, int ld, const double* __restrict__ r,
                                            const T* __restrict__ b) {
    double s = 0.0;
#pragma unroll 4
    for (int j = (threadIdx.x & 31) * 2; j < ld; j += 64) {
        double a[2];
        *reinterpret_cast<uint4*>(a) = __ldg(reinterpret_cast<const uint4*>(r + j));
#pragma unroll
        for (int v = 0; v < 2; v++) s += a[v] * (j + v < n ? (double)__ldg(b + j + v) : 0.0);
    }
    return warp_sum(s);
}

// x = B b, one warp a row
template <typename T>
__global__ void __launch_bounds__(128)
k_dense_mv(int n, int ld, const double* __restrict__ B, const T* __restrict__ b, T* __restrict__ x) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= n) return;
    const double s = dense_row(n, ld, B + (size_t)row * ld, b);
    if ((threadIdx.x & 31) == 0) x[row] = (T)s;
}

// X = B b for k interleaved columns (entry (j, c) at j k + c): one warp a row
// and kDenseCols of its columns (blockIdx.y), the row of B read once for them.
constexpr int kDenseCols = 8;
template <typename T>
__global__ void __launch_bounds__(128)
k_dense_mm(int n, int ld, const double* __restrict__ B, int k, const T* __restrict__ b,
           T* __restrict__ x) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int c0 = blockIdx.y * kDenseCols;
    if (row >= n) return;
    const double* r = B + (size_t)row * ld;
    double s[kDenseCols] = {};
#pragma unroll 2
    for (int j = lane; j < n; j += 32) {
        const double a = __ldg(r + j);
        T v[kDenseCols];
#pragma unroll
        for (int c = 0; c < kDenseCols; c++) v[c] = c0 + c < k ? __ldg(b + (size_t)j * k + c0 + c) : T(0);
#pragma unroll
        for (int c = 0; c < kDenseCols; c++) s[c] += a * (double)v[c];
    }
#pragma unroll
    for (int c = 0; c < kDenseCols; c++) {
        const double t = warp_sum(s[c]);
        if (lane == 0 && c0 + c < k) x[(size_t)row * k + c0 + c] = (T)t;
    }
}

// ------------------------------------------------------- forming B (FP64) --
// out (n x m, row-major) = the transpose of a column-major n x n matrix
static __global__ void k_dense_from_inverse(int n, const double* __restrict__ inv, double* out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (c < n) out[(size_t)i * n + c] = inv[(size_t)c * n + i];
}

// M = I - A D, one warp a row (M zeroed before; a thread a row waited for its
// entries one by one).  The adds are atomic for a row that names a column
// twice; where none does, as in every product matrix, each entry has one.
template <typename T>
__global__ void k_dense_first_residual(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                       const double* __restrict__ cv, const T* __restrict__ d,
                                       double* M) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    double* row = M + (size_t)i * n;
    if (lane == 0) row[i] = 1.0;
    __syncwarp();
    for (int j = rp[i] + lane; j < rp[i + 1]; j += 32) {
        const int c = ci[j];
        atomicAdd(row + c, -(cv[j] * (double)d[c]));
    }
}

// M = the CSR matrix, dense with m columns (M zeroed before)
static __global__ void k_dense_copy(int n, int m, const int* __restrict__ rp,
                                    const int* __restrict__ ci, const double* __restrict__ cv,
                                    double* M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int j = rp[i]; j < rp[i + 1]; j++) M[(size_t)i * m + ci[j]] += cv[j];
}

// Y = S X for CSR S (rows of Y one a blockIdx.y, m columns), then
// MODE 0: out = Y;  1: out = diag(d) + Y;  2: out = X + diag(d) (I - Y),
// S square.
template <int MODE, typename T>
__global__ void __launch_bounds__(256)
k_dense_spmm(int m, const int* __restrict__ rp, const int* __restrict__ ci,
             const double* __restrict__ cv, const double* __restrict__ X, const T* __restrict__ d,
             double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (c >= m) return;
    double s = 0.0;
    const int e = rp[i + 1];
#pragma unroll 4
    for (int j = rp[i]; j < e; j++) s += cv[j] * X[(size_t)ci[j] * m + c];
    if (MODE == 1) s += c == i ? (double)d[i] : 0.0;
    if (MODE == 2) s = X[(size_t)i * m + c] + (double)d[i] * ((c == i ? 1.0 : 0.0) - s);
    out[(size_t)i * m + c] = s;
}

// C (n x m) = A (n x n) B (n x m), FP64, row-major: 32 x 64 tiles, 256
// threads of 2 x 4 entries, 16 of the inner dimension a step.
static __global__ void __launch_bounds__(256)
k_dense_gemm(int n, int m, const double* __restrict__ A, const double* __restrict__ B,
             double* __restrict__ C) {
    __shared__ double sa[16][33], sb[16][64];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 64;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    double acc[2][4] = {};
    for (int k0 = 0; k0 < n; k0 += 16) {
        for (int t = threadIdx.x; t < 32 * 16; t += 256) {
            const int r = t / 16, k = t % 16;
            sa[k][r] = r0 + r < n && k0 + k < n ? A[(size_t)(r0 + r) * n + k0 + k] : 0.0;
        }
        for (int t = threadIdx.x; t < 16 * 64; t += 256) {
            const int k = t / 64, c = t % 64;
            sb[k][c] = k0 + k < n && c0 + c < m ? B[(size_t)(k0 + k) * m + c0 + c] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double a0 = sa[k][ty * 2], a1 = sa[k][ty * 2 + 1];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const double b = sb[k][tx + 16 * q];
                acc[0][q] += a0 * b;
                acc[1][q] += a1 * b;
            }
        }
        __syncthreads();
    }
    for (int p = 0; p < 2; p++)
        for (int q = 0; q < 4; q++) {
            const int r = r0 + ty * 2 + p, c = c0 + tx + 16 * q;
            if (r < n && c < m) C[(size_t)r * m + c] = acc[p][q];
        }
}

// B with its rows padded to ld
static __global__ void k_dense_store(int n, int ld, const double* __restrict__ in,
                                     double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (c < ld) out[(size_t)i * ld + c] = c < n ? in[(size_t)i * n + c] : 0.0;
}

}  // namespace rb
