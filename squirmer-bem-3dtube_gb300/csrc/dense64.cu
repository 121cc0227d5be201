// dense64.cu -- FP64 GEMM, certified no-exchange blocked LU with a partial-
// pivoting fallback, and blocked LU solves (the SQBEM_FP64 path; replaces the
// reference's dgemm_/dgetrf_/dgetrs_/dgesv_, src/utils/linalg.hpp:17-78).
//
// GB300 executes FP64 at roughly 1 TFLOP/s (CUDA-core DFMA and DMMA alike).  Large
// products therefore run as digit products on the BF16 tensor cores with FP64
// results (oz_gemm.cu); what stays on the FP64 pipe is the work around them: the
// panels of the LU, and products with a few columns.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "dense.cuh"
#include "oz_gemm.cuh"

namespace cg = cooperative_groups;

namespace sqbem {

// ---------------------------------------------------------------- GEMM
constexpr int GB_M = 64, GB_N = 64, GB_K = 16;

template <bool TA, bool TB>
__global__ void __launch_bounds__(256) dgemm_kernel(int M, int N, int K, double alpha, const double* __restrict__ A,
                                                    long long lda, const double* __restrict__ B, long long ldb,
                                                    double beta, double* __restrict__ C, long long ldc) {
    __shared__ double As[GB_K][GB_M + 1];
    __shared__ double Bs[GB_K][GB_N + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.x * GB_M, n0 = blockIdx.y * GB_N;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    for (int k0 = 0; k0 < K; k0 += GB_K) {
#pragma unroll
        for (int r = 0; r < (GB_M * GB_K) / 256; ++r) {
            const int e = tid + r * 256;
            const int m = TA ? e / GB_K : e % GB_M;
            const int k = TA ? e % GB_K : e / GB_M;
            const int gm = m0 + m, gk = k0 + k;
            double v = 0.0;
            if (gm < M && gk < K) v = TA ? A[gk + gm * lda] : A[gm + gk * lda];
            As[k][m] = v;
        }
#pragma unroll
        for (int r = 0; r < (GB_N * GB_K) / 256; ++r) {
            const int e = tid + r * 256;
            const int n = TB ? e % GB_N : e / GB_K;
            const int k = TB ? e / GB_N : e % GB_K;
            const int gn = n0 + n, gk = k0 + k;
            double v = 0.0;
            if (gk < K && gn < N) v = TB ? B[gn + gk * ldb] : B[gk + gn * ldb];
            Bs[k][n] = v;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GB_K; ++k) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[k][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int gn = n0 + ty + 16 * j;
        if (gn >= N) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int gm = m0 + tx + 16 * i;
            if (gm >= M) continue;
            double* c = C + gm + gn * ldc;
            *c = beta == 0.0 ? alpha * acc[i][j] : fma(alpha, acc[i][j], beta * *c);
        }
    }
}

// Products with up to 8 columns (right-hand sides).  Reading A is the work: 8 bytes
// per 2 n FP64 operations, so above n = 2 the FP64 pipe bounds it.  The 64 x 64
// tiles above put such a product on a handful of CTAs, each walking all of K.
struct Strides {
    long long a = 0, b = 0, c = 0;  // from one matrix of a batch (blockIdx.y) to the next
};

// C = alpha A B + beta C, A column-major: 32 rows per CTA, 8 warps split K, each
// lane one row (a column's 32 rows are one 256-byte read).
template <int N>
__global__ void __launch_bounds__(256) skinny_n_kernel(int M, int K, double alpha, const double* __restrict__ A,
                                                       long long lda, const double* __restrict__ B, long long ldb,
                                                       double beta, double* __restrict__ C, long long ldc, Strides bs) {
    __shared__ double part[8][N][32];
    A += blockIdx.y * bs.a;
    B += blockIdx.y * bs.b;
    C += blockIdx.y * bs.c;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m = blockIdx.x * 32 + lane;
    double acc[N];
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = 0.0;
    if (m < M) {
#pragma unroll 8
        for (int k = w; k < K; k += 8) {
            const double a = A[m + k * lda];
#pragma unroll
            for (int j = 0; j < N; ++j) acc[j] = fma(a, B[k + j * ldb], acc[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) part[w][j][lane] = acc[j];
    __syncthreads();
    if (m >= M) return;
    for (int j = w; j < N; j += 8) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += part[q][j][lane];
        double* c = C + m + j * ldc;
        *c = beta == 0.0 ? alpha * s : fma(alpha, s, beta * *c);
    }
}

// C = alpha A^T B + beta C: a warp per row of C, the lanes along K (contiguous in A).
template <int N>
__global__ void __launch_bounds__(256) skinny_t_kernel(int M, int K, double alpha, const double* __restrict__ A,
                                                       long long lda, const double* __restrict__ B, long long ldb,
                                                       double beta, double* __restrict__ C, long long ldc, Strides bs) {
    A += blockIdx.y * bs.a;
    B += blockIdx.y * bs.b;
    C += blockIdx.y * bs.c;
    const int lane = threadIdx.x & 31, m = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (m >= M) return;
    double acc[N];
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = 0.0;
    const double* a = A + m * lda;
#pragma unroll 4
    for (int k = lane; k < K; k += 32) {
        const double x = a[k];
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] = fma(x, B[k + j * ldb], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
#pragma unroll
    for (int j = 0; j < N; ++j)
        if (lane == j) {
            double* c = C + m + j * ldc;
            *c = beta == 0.0 ? alpha * acc[j] : fma(alpha, acc[j], beta * *c);
        }
}

// The same with 8 rows per CTA and 32 slices of K: a 256 x 256 block inverse on 32 SMs instead
// of 8 (18 us before).
template <int N>
__global__ void __launch_bounds__(256) skinny_n8_kernel(int M, int K, double alpha, const double* __restrict__ A,
                                                        long long lda, const double* __restrict__ B, long long ldb,
                                                        double beta, double* __restrict__ C, long long ldc, Strides bs) {
    __shared__ double part[8][N][8];
    A += blockIdx.y * bs.a;
    B += blockIdx.y * bs.b;
    C += blockIdx.y * bs.c;
    const int r = threadIdx.x & 7, q = threadIdx.x >> 3, w = threadIdx.x >> 5;
    const int m = blockIdx.x * 8 + r;
    double acc[N];
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = 0.0;
    if (m < M) {
#pragma unroll 8
        for (int k = q; k < K; k += 32) {
            const double a = A[m + k * lda];
#pragma unroll
            for (int j = 0; j < N; ++j) acc[j] = fma(a, B[k + j * ldb], acc[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 8);
        acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
        if ((threadIdx.x & 31) < 8) part[w][j][r] = acc[j];
    }
    __syncthreads();
    if (threadIdx.x < 8 * N) {
        const int j = threadIdx.x >> 3;
        if (m >= M) return;
        double s = 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) s += part[u][j][r];
        double* c = C + m + j * ldc;
        *c = beta == 0.0 ? alpha * s : fma(alpha, s, beta * *c);
    }
}

template <int N>
static void skinny(bool ta, int M, int K, double alpha, const double* A, long long lda, const double* B, long long ldb,
                   double beta, double* C, long long ldc, cudaStream_t st, int batch, Strides bs) {
    const double fl = 2.0 * batch * M * N * K, by = batch * 8.0 * ((double)M * K + (double)K * N + (beta == 0.0 ? 1.0 : 2.0) * M * N);
    if (ta)
        TIMED_LAUNCH("dgemm", fl, by, skinny_t_kernel<N>, dim3(ceil_div(M, 8), batch), 256, 0, st, M, K, alpha, A, lda, B,
                     ldb, beta, C, ldc, bs);
    else if ((long long)M * batch <= 152 * 8 * 2)  // 32-row CTAs would leave most SMs idle
        TIMED_LAUNCH("dgemm", fl, by, skinny_n8_kernel<N>, dim3(ceil_div(M, 8), batch), 256, 0, st, M, K, alpha, A, lda, B,
                     ldb, beta, C, ldc, bs);
    else
        TIMED_LAUNCH("dgemm", fl, by, skinny_n_kernel<N>, dim3(ceil_div(M, 32), batch), 256, 0, st, M, K, alpha, A, lda, B,
                     ldb, beta, C, ldc, bs);
}

void gemm64_few(bool ta, int M, int N, int K, double alpha, const double* A, long long lda, const double* B,
                long long ldb, double beta, double* C, long long ldc, cudaStream_t st, int batch, long long sa,
                long long sb, long long sc) {
    const Strides bs{sa, sb, sc};
    switch (N) {
        case 1: return skinny<1>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 2: return skinny<2>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 3: return skinny<3>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 4: return skinny<4>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 5: return skinny<5>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 6: return skinny<6>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 7: return skinny<7>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        case 8: return skinny<8>(ta, M, K, alpha, A, lda, B, ldb, beta, C, ldc, st, batch, bs);
        default: fail(SQBEM_ERR_ARG, "gemm64_few: %d columns", N);
    }
}

// C (m x 6) = A K for the rigid-body map K of np panels (swimmer.hpp:224-231): row 3p + b of K
// is a unit vector and r_p x e_b, so a panel's three columns take 9 FP64 operations where
// the dense product takes 18.  32 rows per CTA, 8 warps split the panels.
__global__ void __launch_bounds__(256) rigid64_kernel(int m, int np, const double* __restrict__ A, long long lda,
                                                      const double* __restrict__ r, double* __restrict__ C,
                                                      long long ldc) {
    __shared__ double part[8][6][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    double c[6] = {0, 0, 0, 0, 0, 0};
    if (i < m) {
#pragma unroll 4
        for (int p = w; p < np; p += 8) {
            const double* a = A + i + 3LL * p * lda;
            const double a0 = a[0], a1 = a[lda], a2 = a[2 * lda];
            const double rx = r[3 * p], ry = r[3 * p + 1], rz = r[3 * p + 2];
            c[0] += a0;
            c[1] += a1;
            c[2] += a2;
            c[3] = fma(a2, ry, fma(-a1, rz, c[3]));
            c[4] = fma(a0, rz, fma(-a2, rx, c[4]));
            c[5] = fma(a1, rx, fma(-a0, ry, c[5]));
        }
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) part[w][j][lane] = c[j];
    __syncthreads();
    if (w >= 6 || i >= m) return;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += part[q][w][lane];
    C[i + w * ldc] = s;
}

void rigid64(int m, int np, const double* A, long long lda, const double* r, double* C, long long ldc, cudaStream_t st) {
    if (m <= 0) return;
    TIMED_LAUNCH("dgemm", 9.0 * m * np, 24.0 * m * np, rigid64_kernel, ceil_div(m, 32), 256, 0, st, m, np, A, lda, r, C,
                 ldc);
}

// The digit products need about 65 us whatever the size (the scales, two splits, a tile's 36
// products and read-outs), in which the FP64 pipe does 6e7 operations; and a tile of
// 128 x 128 with a K below 64 costs more to read out than to multiply.
constexpr double PIPE_OPS = 6e7;
static bool use_tensor(int M, int N, int K, const int* err) {
    return err && K >= 64 && M >= 64 && N >= 64 && 2.0 * M * N * K > PIPE_OPS;
}

void gemm64(bool ta, bool tb, int M, int N, int K, double alpha, const double* A, long long lda, const double* B,
            long long ldb, double beta, double* C, long long ldc, cudaStream_t st, int* err) {
    if (M <= 0 || N <= 0) return;
    if (K <= 0) {
        // C = beta C
        if (beta == 1.0) return;
        K = 0;
    }
    if (N <= SK_N && !tb) return gemm64_few(ta, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, st);
    if (use_tensor(M, N, K, err)) {
        oz_product(A, ta ? lda : 1, ta ? 1 : lda, B, tb ? 1 : ldb, tb ? ldb : 1, M, N, K, alpha, beta, C, ldc, err, st);
        return;
    }
    dim3 grid(ceil_div(M, GB_M), ceil_div(N, GB_N));
    const double fl = 2.0 * M * N * K;
    const double by = 8.0 * ((double)M * K + (double)K * N + (beta == 0.0 ? 1.0 : 2.0) * M * N);
    if (!ta && !tb)
        TIMED_LAUNCH("dgemm", fl, by, (dgemm_kernel<false, false>), grid, 256, 0, st, M, N, K, alpha, A, lda, B, ldb,
                     beta, C, ldc);
    else if (ta && !tb)
        TIMED_LAUNCH("dgemm", fl, by, (dgemm_kernel<true, false>), grid, 256, 0, st, M, N, K, alpha, A, lda, B, ldb,
                     beta, C, ldc);
    else if (!ta && tb)
        TIMED_LAUNCH("dgemm", fl, by, (dgemm_kernel<false, true>), grid, 256, 0, st, M, N, K, alpha, A, lda, B, ldb,
                     beta, C, ldc);
    else
        TIMED_LAUNCH("dgemm", fl, by, (dgemm_kernel<true, true>), grid, 256, 0, st, M, N, K, alpha, A, lda, B, ldb,
                     beta, C, ldc);
}

void WaitError::check() {
    if (!w.get()) return;
    int h = 0;
    w.download(&h, 1);
    CUDA_CHECK(cudaStreamSynchronize(w.st));
    if (h) fail(SQBEM_ERR_TIMEOUT, "a bounded wait in the FP64 tensor-core product expired");
}

int* WaitError::get(cudaStream_t st) {
    if (!w.get()) {
        w.alloc(1, st);
        w.zero();
    }
    return w.get();
}

// ---------------------------------------------------------------- small helpers
__global__ void copy_kernel(const double* __restrict__ s, long long lds, double* __restrict__ d, long long ldd, int rows,
                            int cols) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)rows * cols) return;
    const int r = (int)(t % rows), c = (int)(t / rows);
    d[r + c * ldd] = s[r + c * lds];
}

void copy_matrix64(const double* src, long long lds, double* dst, long long ldd, int rows, int cols, cudaStream_t st) {
    if (rows <= 0 || cols <= 0) return;
    LAUNCH(copy_kernel, ceil_div((long long)rows * cols, 256), 256, 0, st, src, lds, dst, ldd, rows, cols);
}

// non-negative doubles order like their bit patterns
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
    atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

__global__ void max_abs_kernel(const double* __restrict__ A, long long lda, int rows, int cols, double* out) {
    double m = 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)rows * cols;
         t += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(t % rows), c = (int)(t / rows);
        m = fmax(m, fabs(A[r + c * lda]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, m);
}

void max_abs64(const double* A, long long lda, int rows, int cols, double* out, cudaStream_t st) {
    CUDA_CHECK(cudaMemsetAsync(out, 0, sizeof(double), st));
    if (rows <= 0 || cols <= 0) return;
    LAUNCH(max_abs_kernel, std::min(ceil_div((long long)rows * cols, 256), 152 * 8), 256, 0, st, A, lda, rows, cols,
           out);
}

// ---------------------------------------------------------------- panels of the LU
// A panel of HB = 128 columns is factored in steps of PB = 32 columns:
//   diag      the 32 x 32 diagonal block (one CTA);
//   trsm32    below it L21 = A21 U11^{-1}, right of it U12 = L11^{-1} A12 within
//             the panel, 16 rows or columns per CTA;
//   update32  the rest of the panel, A22 -= L21 U12; the CTA of the next diagonal
//             block updates only that block and factors it at once.
// An FP64 warp instruction occupies its SM quarter's pipe for 64 to 76 cycles, whether its
// lanes are needed or not and whether the next one depends on it or not.  So the kernels
// here count warp instructions: work spread over many CTAs of four warps, no FP64 comparisons
// (integers order like the magnitudes), no per-step divisions.
constexpr int PB = 32, HB = 128;

// 1/x from the hardware's approximate reciprocal y (relative error e = 1 - x y about 2^-20):
// 1/x = y / (1 - e) = y (1 + e + e^2 + ..), cut after e^2, so 2^-60 and the rounding: within one
// unit in the last place of the division.  Three FP64 operations where the full division (430
// cycles) is on the factorisation's serial chain.
__device__ __forceinline__ double recip(double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    if (e < 64 || e > 1980) return 1.0 / x;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double d = fma(-x, y, 1.0);
    return fma(y, fma(d, d, d), y);
}

__global__ void recip_kernel(int n, const double* __restrict__ x, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = recip(x[i]);
}

void recip_eval(int n, const double* x, double* y, cudaStream_t st) {
    if (n > 0) LAUNCH(recip_kernel, ceil_div(n, 256), 256, 0, st, n, x, y);
}

// |x| > |piv|, as a pivot search sees it (bit 0), or x not finite (bit 1); piv by its bits
// without the sign
__device__ __forceinline__ int exceeds(double x, long long piv) {
    const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
    return b > piv ? (b < 0x7ff0000000000000ll ? 1 : 2) : 0;
}

// LU without exchanges of a 32 x 32 block by 128 threads, lane = row, v[u] = column w + 4 u of
// warp w; the first kb columns are factored (the rest of the block: identity).  flag bit 0
// if a multiplier exceeds 1 in magnitude, bit 1 on a zero / non-finite pivot.  The
// finished columns go to out (leading dimension ldo; kb rows and columns).
// Column j belongs to warp j & 3: it publishes the column's multipliers through shared
// memory and a barrier that only the other warps wait on, before its own updates of the step.
__device__ void lu32(double (&v)[8], double (*lc)[PB], int kb, double* out, long long ldo, int* flag) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int bad = 0;
    auto publish = [&](int j) {  // by the warp that holds column j in v[0]
        const double piv = __shfl_sync(0xffffffffu, v[0], j);
        const long long pb = __double_as_longlong(piv) & 0x7fffffffffffffffll;
        if (pb == 0 || pb >= 0x7ff0000000000000ll) bad |= 2;
        const double l = v[0] * recip(piv);
        if (lane > j) {
            bad |= exceeds(v[0], pb);
            v[0] = l;
        }
        lc[j & 3][lane] = lane > j ? l : 0.0;
        __threadfence_block();
        asm volatile("barrier.cta.arrive %0, 128;" ::"r"(1 + (j & 3)) : "memory");
    };
    if (w == 0) publish(0);
    for (int t = 0; 4 * t < kb; ++t) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int j = 4 * t + s;
            if (w != s) asm volatile("barrier.cta.sync %0, 128;" ::"r"(1 + s) : "memory");
            const double l = lc[s][lane];
            if (w > s) v[0] = fma(-l, __shfl_sync(0xffffffffu, v[0], j), v[0]);
            if (s < 3 && w == s + 1) publish(j + 1);
#pragma unroll
            for (int u = 1; u < 8; ++u) {
                if (4 * (t + u) < kb) v[u] = fma(-l, __shfl_sync(0xffffffffu, v[u], j), v[u]);
                if (u == 1 && s == 3 && w == 0 && j + 1 < PB) {  // column j + 1 is next in line: v[1] of warp 0
                    const double keep = v[0];
                    v[0] = v[1];
                    publish(j + 1);
                    v[1] = v[0];
                    v[0] = keep;
                }
            }
        }
        if (lane < kb && w + 4 * t < kb) out[lane + (w + 4 * t) * ldo] = v[0];
#pragma unroll
        for (int u = 0; u < 7; ++u) v[u] = v[u + 1];
    }
    // the last publication has no readers: take the barrier back to its start
    if (((kb + 3) & ~3) < PB && w != 0) asm volatile("barrier.cta.sync %0, 128;" ::"r"(1) : "memory");
    if (bad) atomicOr(flag, bad);
}

__global__ void __launch_bounds__(128) lu_diag_kernel(double* A, long long lda, int kb, int* flag) {
    __shared__ double lc[4][PB];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int c = w + 4 * u;
        v[u] = lane < kb && c < kb ? A[lane + c * lda] : (lane == c ? 1.0 : 0.0);
    }
    lu32(v, lc, kb, A, lda, flag);
}

// A points at the factored kb x kb diagonal block (kb <= 32); m rows below it, w columns
// right of it.  CTAs 0 .. ceil(m / 16) - 1 take rows, the others columns; eight lanes
// share a row (column), each holding every eighth of its 32 entries.  A row's substitution
// carries y_j = x_j u_jj and the scaled factor u_jk / u_jj, so that the divisions come
// once at the end.
__global__ void __launch_bounds__(128) lu_trsm32_kernel(double* A, long long lda, int kb, int m, int w, int* flag) {
    __shared__ double t[PB][PB + 1];  // rows: U11 by [j][k] over u_jj; columns: L11^T by [j][i]; 0 for k <= j
    __shared__ double rd[PB];
    __shared__ long long ad[PB];
    const int nrow = (m + 15) >> 4;
    const bool rows = (int)blockIdx.x < nrow;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, q = lane & 7;
    const int idx = (rows ? blockIdx.x : blockIdx.x - nrow) * 16 + (threadIdx.x >> 3);
    const bool in = idx < (rows ? m : w);
    // entry k of this row (column)
    double* const p = rows ? A + kb + idx : A + (kb + idx) * lda;
    const long long s = rows ? lda : 1;
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = in && q + 8 * u < kb ? p[(q + 8 * u) * s] : 0.0;
    double e[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int c = g + 4 * u;
        e[u] = lane < kb && c < kb ? A[lane + c * lda] : (lane == c ? 1.0 : 0.0);
    }
    double piv = 1.0;  // of column lane, where this warp holds it
#pragma unroll
    for (int u = 0; u < 8; ++u)
        if (lane == g + 4 * u) piv = e[u];
    piv = (lane & 3) == g ? piv : 1.0;
    const double rp = recip(piv);
    if ((lane & 3) == g) {
        rd[lane] = rp;
        ad[lane] = __double_as_longlong(piv) & 0x7fffffffffffffffll;
    }
    __syncthreads();
    if (rows) {
        const double r = rd[lane];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[lane][g + 4 * u] = g + 4 * u > lane ? e[u] * r : 0.0;
    } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) t[g + 4 * u][lane] = lane > g + 4 * u ? e[u] : 0.0;
    }
    __syncthreads();
    int bad = 0;
#pragma unroll
    for (int j = 0; j < PB; ++j) {
        const double y = __shfl_sync(0xffffffffu, v[j >> 3], (lane & ~7) | (j & 7));
        if (rows) bad |= exceeds(y, ad[j]);
#pragma unroll
        for (int u = j >> 3; u < 4; ++u)
            if (j != 8 * u + 7) v[u] = fma(-y, t[j][q + 8 * u], v[u]);
    }
    if (!in) return;
    if (bad) atomicOr(flag, bad);
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (q + 8 * u < kb) p[(q + 8 * u) * s] = rows ? v[u] * rd[q + 8 * u] : v[u];
}

// A22 -= L21 U12 for the m rows and w <= 96 columns past a full 32 x 32 diagonal block
// at A.  The first cluster of four CTAs takes the next diagonal block (nb x nb), eight
// columns each (one SM alone took 10 us for it), and its first CTA factors it; the other
// CTAs 16 rows each, without that block's columns in its rows.
constexpr int UPD_CL = 4;
__global__ void __cluster_dims__(UPD_CL, 1, 1) __launch_bounds__(128)
    lu_update32_kernel(double* A, long long lda, int m, int w, int nb, int* flag) {
    __shared__ double L[PB][PB + 1];      // [k][row]
    __shared__ double U[PB][3 * PB + 1];  // [k][column]
    __shared__ double lc[4][PB];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (blockIdx.x < UPD_CL) {
        cg::cluster_group cl = cg::this_cluster();
        const int cb = 8 * blockIdx.x + 2 * wp;
        double acc[2];
#pragma unroll
        for (int u = 0; u < 8; ++u) L[wp + 4 * u][lane] = lane < nb ? A[PB + lane + (wp + 4 * u) * lda] : 0.0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = cb + u;
            U[lane][c] = c < nb ? A[lane + (PB + c) * lda] : 0.0;
            acc[u] = lane < nb && c < nb ? A[PB + lane + (PB + c) * lda] : (lane == c ? 1.0 : 0.0);
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < PB; ++k) {
            const double l = L[k][lane];
#pragma unroll
            for (int u = 0; u < 2; ++u) acc[u] = fma(-l, U[k][cb + u], acc[u]);
        }
        // gathered in the first CTA's U, by [column][row]
        cl.sync();
        double (*const G)[PB + 1] = reinterpret_cast<double (*)[PB + 1]>(cl.map_shared_rank(&U[0][0], 0));
#pragma unroll
        for (int u = 0; u < 2; ++u) G[cb + u][lane] = acc[u];
        cl.sync();
        if (blockIdx.x != 0) return;
        double v[8];
        const double (*const g)[PB + 1] = reinterpret_cast<const double (*)[PB + 1]>(&U[0][0]);
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = g[wp + 4 * u][lane];
        lu32(v, lc, nb, A + PB + PB * lda, lda, flag);
        return;
    }
    const int row = (blockIdx.x - UPD_CL) * 16 + (lane & 15), g = wp * 2 + (lane >> 4);
    const int c0 = row < nb ? nb : 0;
#pragma unroll
    for (int k = g; k < PB; k += 8) L[k][lane & 15] = row < m ? A[PB + row + k * lda] : 0.0;
#pragma unroll 8
    for (int c = wp; c < w; c += 4) U[lane][c] = A[lane + (PB + c) * lda];
    double acc[12];
#pragma unroll
    for (int u = 0; u < 12; ++u) {
        const int c = g + 8 * u;
        acc[u] = row < m && c < w ? A[PB + row + (PB + c) * lda] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < PB; ++k) {
        const double l = L[k][lane & 15];
#pragma unroll
        for (int u = 0; u < 12; ++u)
            if (8 * u < w) acc[u] = fma(-l, U[k][g + 8 * u], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 12; ++u) {
        const int c = g + 8 * u;
        if (row < m && c >= c0 && c < w) A[PB + row + (PB + c) * lda] = acc[u];
    }
}

// X <- L^{-1} X or U^{-1} X for the diagonal blocks of a factored matrix, C columns per CTA
// (one where a single block's latency counts, two for all blocks of a matrix), a thread per row, one barrier per step; warps whose rows are finished skip the
// step's FMAs.  The triangle's column for a step does not depend on the steps before, so
// eight are loaded ahead (waiting for each one's L2 round trip took 64 us for 128 steps).
//   lu_lower_kernel    X = columns of the matrix right of block A (in place)
//   lu_inverse_kernel  X = identity: the inverse of block blockIdx.x's triangle, column-major
//                      with leading dimension LU_NB, zero padded.
constexpr int INV_AHEAD = 8;
template <bool LOWER, int INV_C>
__device__ void tri_solve(const double* a, long long lda, int rows, int first, int steps, double rd,
                          double (&r)[INV_C], double (*x)[INV_C]) {
    const int i = threadIdx.x, d = LOWER ? 1 : -1;
    auto entry = [&](int s) {
        const int j = first + d * s;
        return s < steps && i < rows && (LOWER ? i > j : i < j) ? a[i + (long long)j * lda] : 0.0;
    };
    double t[INV_AHEAD];
#pragma unroll
    for (int u = 0; u < INV_AHEAD; ++u) t[u] = entry(u);
    for (int s0 = 0; s0 < steps; s0 += INV_AHEAD) {
        double nx[INV_AHEAD];
#pragma unroll
        for (int u = 0; u < INV_AHEAD; ++u) nx[u] = entry(s0 + INV_AHEAD + u);
#pragma unroll
        for (int u = 0; u < INV_AHEAD; ++u) {
            if (s0 + u >= steps) break;
            const int j = first + d * (s0 + u);
            if (i == j)
#pragma unroll
                for (int c = 0; c < INV_C; ++c) {
                    if (!LOWER) r[c] *= rd;
                    x[j][c] = r[c];
                }
            __syncthreads();
            if (LOWER ? (i | 31) > j : (i & ~31) < j)
#pragma unroll
                for (int c = 0; c < INV_C; ++c) r[c] = fma(-t[u], x[j][c], r[c]);
        }
#pragma unroll
        for (int u = 0; u < INV_AHEAD; ++u) t[u] = nx[u];
    }
}

constexpr int LOWER_C = 1;
__global__ void __launch_bounds__(HB) lu_lower_kernel(double* A, long long lda, int w) {
    constexpr int INV_C = LOWER_C;
    __shared__ double x[HB][INV_C];
    const int i = threadIdx.x, c0 = blockIdx.x * INV_C;
    double* X = A + (long long)(HB + c0) * lda + i;
    double r[INV_C];
#pragma unroll
    for (int c = 0; c < INV_C; ++c) r[c] = c0 + c < w ? X[c * lda] : 0.0;
    tri_solve<true, INV_C>(A, lda, HB, 0, HB, 1.0, r, x);
#pragma unroll
    for (int c = 0; c < INV_C; ++c)
        if (c0 + c < w) X[c * lda] = r[c];
}

template <int INV_C>
__global__ void __launch_bounds__(LU_NB) lu_inverse_kernel(const double* __restrict__ A, long long lda, int n,
                                                           bool upper, double* __restrict__ inv) {
    __shared__ double x[LU_NB][INV_C];
    const int k0 = blockIdx.x * LU_NB, kb = min(LU_NB, n - k0), i = threadIdx.x;
    const int c0 = blockIdx.y * INV_C;
    const double* a = A + k0 + (long long)k0 * lda;
    double r[INV_C];
#pragma unroll
    for (int c = 0; c < INV_C; ++c) r[c] = i == c0 + c && i < kb ? 1.0 : 0.0;
    if (c0 < kb) {
        const int last = min(kb, c0 + INV_C) - 1;
        if (!upper) tri_solve<true, INV_C>(a, lda, kb, c0, kb - c0, 1.0, r, x);
        else tri_solve<false, INV_C>(a, lda, kb, last, last + 1, i < kb ? recip(a[i + (long long)i * lda]) : 0.0, r, x);
    }
    double* o = inv + (long long)blockIdx.x * LU_NB * LU_NB + i;
#pragma unroll
    for (int c = 0; c < INV_C; ++c) o[(c0 + c) * LU_NB] = i < kb ? r[c] : 0.0;
}

// ---------------------------------------------------------------- pivoted fallback
// Column j of an unblocked right-looking LU with partial pivoting (dgetf2 order).
__global__ void __launch_bounds__(1024) pivot_kernel(const double* A, long long lda, int n, int j, int* ipiv, int* flag) {
    __shared__ double bv[32];
    __shared__ int bi[32];
    double best = -1.0;
    int bidx = n;
    for (int i = j + threadIdx.x; i < n; i += blockDim.x) {
        const double v = fabs(A[i + j * lda]);
        if (v > best) { best = v; bidx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
        if (ov > best || (ov == best && oi < bidx)) { best = ov; bidx = oi; }
    }
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = bidx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            if (bv[w] > best || (bv[w] == best && bi[w] < bidx)) { best = bv[w]; bidx = bi[w]; }
        // first maximum, as idamax; a zero column keeps the diagonal
        if (!(best > 0.0)) { bidx = j; atomicOr(flag, 2); }
        ipiv[j] = bidx;
    }
}

__global__ void swap_rows_kernel(double* A, long long lda, int n, int j, const int* ipiv) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int p = ipiv[j];
    if (c >= n || p == j) return;
    const double t = A[j + c * lda];
    A[j + c * lda] = A[p + c * lda];
    A[p + c * lda] = t;
}

__global__ void rank1_kernel(double* A, long long lda, int n, int j) {
    const int i = j + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int c = j + 1 + blockIdx.y;
    if (i >= n || c >= n) return;
    const double piv = A[j + j * lda];
    if (piv == 0.0) return;
    const double l = A[i + j * lda] / piv;
    A[i + c * lda] = fma(-l, A[j + c * lda], A[i + c * lda]);
}

__global__ void scale_col_kernel(double* A, long long lda, int n, int j) {
    const int i = j + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double piv = A[j + j * lda];
    if (piv != 0.0) A[i + j * lda] = A[i + j * lda] / piv;
}

__global__ void laswp_kernel(double* B, long long ldb, int n, int nrhs, const int* ipiv) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nrhs) return;
    for (int j = 0; j < n; ++j) {
        const int p = ipiv[j];
        if (p != j) {
            const double t = B[j + c * ldb];
            B[j + c * ldb] = B[p + c * ldb];
            B[p + c * ldb] = t;
        }
    }
}

// ---------------------------------------------------------------- LU64
// C = alpha A B + beta C (column-major) by digit products; q: K words of zeros
static void tensor_product(const double* A, long long lda, const double* B, long long ldb, int M, int N, int K,
                           double alpha, double beta, double* C, long long ldc, int* err, cudaStream_t st, int* q) {
    oz_product(A, 1, lda, B, ldb, 1, M, N, K, alpha, beta, C, ldc, err, st, q);
}

// The panel of columns [k0, k0 + kb), kb <= HB, of the n x n matrix, all rows below.
static void factor_panel(double* A, long long ld, int n, int k0, int kb, int* flag, cudaStream_t st) {
    double* A11 = A + k0 + k0 * ld;
    LAUNCH(lu_diag_kernel, 1, 128, 0, st, A11, ld, std::min(PB, kb), flag);
    for (int j = 0; j < kb; j += PB) {
        const int jb = std::min(PB, kb - j), m = n - k0 - j - jb, w = kb - j - jb;
        double* D = A11 + j + j * ld;
        if (m > 0) LAUNCH(lu_trsm32_kernel, ceil_div(m, 16) + ceil_div(w, 16), 128, 0, st, D, ld, jb, m, w, flag);
        if (w > 0) LAUNCH(lu_update32_kernel, UPD_CL * (1 + ceil_div(m, 16 * UPD_CL)), 128, 0, st, D, ld, m, w,
                          std::min(PB, w), flag);
    }
}

// Panels of LU_NB = 256 columns, each as two of 128.  With 256 the trailing update's tiles
// multiply for longer (18 us) than they take to read out, which 128 do not.
static void run_fast(double* A, long long ld, int n, double* Linv, double* Uinv, int* flag, int* err, cudaStream_t st) {
    // the scales of up to three products per panel
    DevBuf<int> scales;
    if (n > HB) {
        scales.alloc(3 * (size_t)LU_NB * ceil_div(n, LU_NB), st);
        scales.zero();
    }
    for (int k0 = 0, b = 0; k0 < n; k0 += LU_NB, ++b) {
        const int kb = std::min(LU_NB, n - k0), n2 = n - k0 - kb, h = std::min(HB, kb), h2 = kb - h;
        double* A11 = A + k0 + k0 * ld;
        int* const q = scales.get() + 3 * (size_t)LU_NB * b;
        factor_panel(A, ld, n, k0, h, flag, st);
        if (h2 > 0) {
            double* right = A11 + h * ld;
            LAUNCH(lu_lower_kernel, ceil_div(h2, LOWER_C), HB, 0, st, A11, ld, h2);
            tensor_product(A11 + h, ld, right, ld, n - k0 - h, h2, h, -1.0, 1.0, right + h, ld, err, st, q);
            factor_panel(A, ld, n, k0 + h, h2, flag, st);
        }
        if (n2 == 0) break;
        double* Li = Linv + (long long)b * LU_NB * LU_NB;
        double* A12 = A + k0 + (k0 + kb) * ld;
        double* A21 = A + (k0 + kb) + k0 * ld;
        double* A22 = A + (k0 + kb) + (k0 + kb) * ld;
        // U12 = L11^{-1} A12
        LAUNCH(lu_inverse_kernel<1>, dim3(1, LU_NB), LU_NB, 0, st, A11, ld, kb, false, Li);
        tensor_product(Li, LU_NB, A12, ld, kb, n2, kb, 1.0, 0.0, A12, ld, err, st, q + LU_NB);
        // A22 -= L21 U12
        tensor_product(A21, ld, A12, ld, n2, n2, kb, -1.0, 1.0, A22, ld, err, st, q + 2 * LU_NB);
    }
    // L^{-1} of the last block, and U^{-1} of all
    const int last = (n - 1) / LU_NB, k0 = last * LU_NB;
    LAUNCH(lu_inverse_kernel<1>, dim3(1, LU_NB), LU_NB, 0, st, A + k0 + k0 * ld, ld, n - k0, false,
           Linv + (long long)last * LU_NB * LU_NB);
    if (last == 0) LAUNCH(lu_inverse_kernel<1>, dim3(1, LU_NB), LU_NB, 0, st, A, ld, n, true, Uinv);
    else LAUNCH(lu_inverse_kernel<2>, dim3(last + 1, LU_NB / 2), LU_NB, 0, st, A, ld, n, true, Uinv);
}

static void run_pivoted(double* A, long long ld, int n, int* ipiv, double* Linv, double* Uinv, int* flag,
                        cudaStream_t st) {
    for (int j = 0; j < n; ++j) {
        LAUNCH(pivot_kernel, 1, 1024, 0, st, A, ld, n, j, ipiv, flag);
        LAUNCH(swap_rows_kernel, ceil_div(n, 256), 256, 0, st, A, ld, n, j, ipiv);
        if (j + 1 < n) {
            LAUNCH(rank1_kernel, dim3(ceil_div(n - j - 1, 256), n - j - 1), 256, 0, st, A, ld, n, j);
            LAUNCH(scale_col_kernel, ceil_div(n - j - 1, 256), 256, 0, st, A, ld, n, j);
        }
    }
    for (int up = 0; up < 2; ++up)
        LAUNCH(lu_inverse_kernel<2>, dim3(ceil_div(n, LU_NB), LU_NB / 2), LU_NB, 0, st, A, ld, n, up != 0,
               up ? Uinv : Linv);
}

// [0]: the certificate, [1]: a bounded wait of the tensor-core products expired
static int read_flag(const int* flag, cudaStream_t st) {
    int h[2] = {0, 0};
    CUDA_CHECK(cudaMemcpyAsync(h, flag, sizeof h, cudaMemcpyDeviceToHost, st));
    count_d2h(sizeof h);
    CUDA_CHECK(cudaStreamSynchronize(st));
    if (h[1]) fail(SQBEM_ERR_TIMEOUT, "LU: a bounded wait in the FP64 tensor-core product expired");
    return h[0];
}

void LU64::factor_inplace(DevBuf<double>&& M, int n_, cudaStream_t st, const char* what) {
    n = n_;
    ld = n_;
    A = std::move(M);
    const int nblk = ceil_div(n, LU_NB);
    Linv.alloc((size_t)nblk * LU_NB * LU_NB, st);
    Uinv.alloc((size_t)nblk * LU_NB * LU_NB, st);
    DevBuf<int> flag(2, st);
    flag.zero();
    DevBuf<double> saved((size_t)n * n, st);
    CUDA_CHECK(cudaMemcpyAsync(saved.get(), A.get(), sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, st));
    run_fast(A.get(), ld, n, Linv.get(), Uinv.get(), flag.get(), flag.get() + 1, st);
    int f = read_flag(flag.get(), st);
    pivoted = false;
    if (f != 0) {
        // certificate failed: redo with row exchanges from the saved matrix
        CUDA_CHECK(cudaMemcpyAsync(A.get(), saved.get(), sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, st));
        ipiv.alloc((size_t)n, st);
        flag.zero();
        run_pivoted(A.get(), ld, n, ipiv.get(), Linv.get(), Uinv.get(), flag.get(), st);
        pivoted = true;
        f = read_flag(flag.get(), st);
        if (f & 2) fail(SQBEM_ERR_SINGULAR, "%s", what);
    }
}

void LU64::factor(const double* M, int n_, long long ldm, cudaStream_t st, const char* what) {
    DevBuf<double> a((size_t)n_ * n_, st);
    copy_matrix64(M, ldm, a.get(), n_, n_, n_, st);
    factor_inplace(std::move(a), n_, st, what);
}

// Few right-hand sides: per block one product with the block's inverse and one update of
// the rows past it, between B and a second buffer (no copies).
static void solve_few(const LU64& lu, int n, double* B, long long ldb, int nrhs, cudaStream_t st) {
    const int nblk = ceil_div(n, LU_NB);
    const long long ld = lu.ld;
    const double* A = lu.A.get();
    // per-call scratch (stream-ordered), so handles sharing one factor on
    // different streams never share a buffer
    DevBuf<double> X((size_t)n * nrhs, st);
    double* x = X.get();
    for (int b = 0; b < nblk; ++b) {  // forward: unit lower L, B -> X
        const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0);
        gemm64(false, false, kb, nrhs, kb, 1.0, lu.Linv.get() + (long long)b * LU_NB * LU_NB, LU_NB, B + k0, ldb, 0.0,
               x + k0, n, st);
        gemm64(false, false, n - k0 - kb, nrhs, kb, -1.0, A + (k0 + kb) + k0 * ld, ld, x + k0, n, 1.0, B + k0 + kb, ldb,
               st);
    }
    for (int b = nblk - 1; b >= 0; --b) {  // backward: U, X -> B
        const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0);
        gemm64(false, false, kb, nrhs, kb, 1.0, lu.Uinv.get() + (long long)b * LU_NB * LU_NB, LU_NB, x + k0, n, 0.0,
               B + k0, ldb, st);
        gemm64(false, false, k0, nrhs, kb, -1.0, A + k0 * ld, ld, B + k0, ldb, 1.0, x, n, st);
    }
}

// Many right-hand sides of a system of one block and few operations: two products with the
// block's inverses, SK_N columns per CTA, all columns at once.  The digits take 130 us for the
// two whatever the size.
static void solve_one_block(const LU64& lu, double* B, long long ldb, int nrhs, cudaStream_t st) {
    const int n = lu.n;
    DevBuf<double> X((size_t)n * nrhs, st);
    auto product = [&](const double* inv, const double* b, long long lb, double* c, long long lc) {
        for (int j = 0, batch; j < nrhs; j += SK_N * batch) {
            batch = std::max(1, std::min(65535, (nrhs - j) / SK_N));
            gemm64_few(false, n, std::min(SK_N, nrhs - j), n, 1.0, inv, LU_NB, b + j * lb, lb, 0.0, c + j * lc, lc, st,
                       batch, 0, SK_N * lb, SK_N * lc);
        }
    };
    product(lu.Linv.get(), B, ldb, X.get(), n);
    product(lu.Uinv.get(), X.get(), n, B, ldb);
}

// Without exchanges the factor of a leading block is the leading block of the factor, and so
// are the inverses of its diagonal blocks.
void LU64::solve_leading(int m, double* B, long long ldb, int nrhs, cudaStream_t st) const {
    if (pivoted || m > n) fail(SQBEM_ERR_ARG, "LU: no factor of the leading block");
    for (int c = 0; c < nrhs; c += SK_N) solve_few(*this, m, B + c * ldb, ldb, std::min(SK_N, nrhs - c), st);
}

void LU64::solve(double* B, long long ldb, int nrhs, cudaStream_t st, int* err) const {
    if (nrhs <= 0 || n == 0) return;
    if (pivoted) LAUNCH(laswp_kernel, ceil_div(nrhs, 128), 128, 0, st, B, ldb, n, nrhs, ipiv.get());
    if (nrhs < 64 || !err) {
        for (int c = 0; c < nrhs; c += SK_N) solve_few(*this, n, B + c * ldb, ldb, std::min(SK_N, nrhs - c), st);
        return;
    }
    if (n <= LU_NB && 2.0 * n * n * nrhs <= PIPE_OPS) return solve_one_block(*this, B, ldb, nrhs, st);
    // many: the block inverses and the updates as tensor-core products
    const int nblk = ceil_div(n, LU_NB);
    DevBuf<int> scales(4 * (size_t)LU_NB * nblk, st);
    scales.zero();
    int* q = scales.get();
    for (int b = 0; b < nblk; ++b) {  // forward: unit lower L
        const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0), n2 = n - k0 - kb;
        tensor_product(Linv.get() + (long long)b * LU_NB * LU_NB, LU_NB, B + k0, ldb, kb, nrhs, kb, 1.0, 0.0, B + k0, ldb,
                       err, st, q);
        q += LU_NB;
        if (n2 > 0)
            tensor_product(A.get() + (k0 + kb) + k0 * ld, ld, B + k0, ldb, n2, nrhs, kb, -1.0, 1.0, B + k0 + kb, ldb, err,
                           st, q);
        q += LU_NB;
    }
    for (int b = nblk - 1; b >= 0; --b) {  // backward: U
        const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0);
        tensor_product(Uinv.get() + (long long)b * LU_NB * LU_NB, LU_NB, B + k0, ldb, kb, nrhs, kb, 1.0, 0.0, B + k0, ldb,
                       err, st, q);
        q += LU_NB;
        if (k0 > 0)
            tensor_product(A.get() + k0 * ld, ld, B + k0, ldb, k0, nrhs, kb, -1.0, 1.0, B, ldb, err, st, q);
        q += LU_NB;
    }
}

}  // namespace sqbem

namespace sqbem {

// B <- P^T applied in reverse exchange order (undoes laswp)
__global__ void laswp_reverse_kernel(double* B, long long ldb, int n, int nrhs, const int* ipiv) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nrhs) return;
    for (int j = n - 1; j >= 0; --j) {
        const int p = ipiv[j];
        if (p != j) {
            const double t = B[j + c * ldb];
            B[j + c * ldb] = B[p + c * ldb];
            B[p + c * ldb] = t;
        }
    }
}

// A^T X = B with P A = L U:  A^T = U^T L^T P, so X = P^T L^{-T} U^{-T} B.
// U^T is lower triangular (forward, block inverses transposed), L^T unit upper
// (backward); the off-diagonal blocks enter as transposed GEMM operands.
void LU64::solve_transpose(double* B, long long ldb, int nrhs, cudaStream_t st) const {
    if (nrhs <= 0 || n == 0) return;
    const int nblk = ceil_div(n, LU_NB);
    DevBuf<double> X((size_t)n * std::min(nrhs, SK_N), st);
    double* x = X.get();
    for (int c = 0; c < nrhs; c += SK_N) {
        const int nr = std::min(SK_N, nrhs - c);
        double* R = B + c * ldb;
        for (int b = 0; b < nblk; ++b) {  // forward with U^T, R -> x: the columns past the block as rows
            const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0);
            gemm64(true, false, kb, nr, kb, 1.0, Uinv.get() + (long long)b * LU_NB * LU_NB, LU_NB, R + k0, ldb, 0.0,
                   x + k0, n, st);
            gemm64(true, false, n - k0 - kb, nr, kb, -1.0, A.get() + k0 + (k0 + kb) * ld, ld, x + k0, n, 1.0,
                   R + k0 + kb, ldb, st);
        }
        for (int b = nblk - 1; b >= 0; --b) {  // backward with L^T (unit), x -> R
            const int k0 = b * LU_NB, kb = std::min(LU_NB, n - k0);
            gemm64(true, false, kb, nr, kb, 1.0, Linv.get() + (long long)b * LU_NB * LU_NB, LU_NB, x + k0, n, 0.0,
                   R + k0, ldb, st);
            gemm64(true, false, k0, nr, kb, -1.0, A.get() + k0, ld, R + k0, ldb, 1.0, x, n, st);
        }
    }
    if (pivoted) LAUNCH(laswp_reverse_kernel, ceil_div(nrhs, 128), 128, 0, st, B, ldb, n, nrhs, ipiv.get());
}

}  // namespace sqbem
