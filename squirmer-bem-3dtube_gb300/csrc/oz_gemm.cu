// oz_gemm.cu -- the kernels of oz_gemm.cuh.
//
// GB300 multiplies FP64 at about 1 TFLOP/s and BF16 on the tensor cores at
// about 1900, so the 36 digit products of an FP64 product still leave room for a
// factor of forty.
//
// One persistent CTA per SM:
//   producer   a warp: bulk copies of the digits' blocks into a ring of 192 KB (the blocks are
//              stored in the order the MMA reads, so the digits a pass needs of one k16 step
//              are one copy per operand);
//   issuers    one warp or two: passes of two weights (d, d + 1), which are the two halves of
//              an accumulator in tensor memory;
//   epilogue   eight warps: the accumulators as integers into 64-bit sums held in registers,
//              the rounding to FP64, C.
// Four passes: weights 0, 1 (digits 0-1) and 2, 3 (digits 0-3) in chunks of 256 k and
// weights 4, 5 in chunks of 160, where every sum is exact (4 * 256 * 2^14 = 2^24, 6 * 160 *
// 2^14 < 2^24); then weights 6, 7 in chunks of 1024 k.  There a sum of weight 6, in units of
// 2^-62 of the product of the largest entries, may reach 2^27 and lose up to 8 units at each of
// its 448 accumulations: 2^-60 of K times that product at most.  (With weights 4, 5 in
// chunks of 1024 too, digits of one sign lost up to 2^-46 of it.)
//   K <= 256 (the panels' updates): tiles of 128 x 64, an accumulator per pass, that of weights
//   4, 5 read out twice for K > 160; the 64-bit sums also take weights 4 and 5 (2^62 at
//   most), and the last pass goes straight into the rounding.
//   K > 256: tiles of 128 x 128, two accumulators; the sums of the leading passes wait in
//   global scratch (L2) for the others, since both sets do not fit in the registers together.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "oz_gemm.cuh"
#include "tc_ptx.cuh"

namespace sqbem {

namespace {

constexpr int TILE = 128;
constexpr int DIGITS = 8;
constexpr int PLANE = TILE * 16 * 2;       // one digit of a 128 x 16 block: 4 KB
constexpr int BLOCK = DIGITS * PLANE;      // 32 KB
constexpr int SMEM_BYTES = 192 * 1024 + 1024 + 256;
constexpr int HI_CHUNK = 16, MID_CHUNK = 10, LO_CHUNK = 64;  // k16 steps between read-outs: passes 0, 1; 2; 3

// Tiles of 128 x TN.  TN = 128 has the widest instructions and suits a long K.  With K <= 256
// a 128 x 128 tile's read-out (20 us) was as long as its multiplication, and with tensor memory
// for two accumulators it ran after it; TN = 64 has all four, so that a tile is multiplied
// during the read-out of the one before, and twice the tiles for products of a few.  Its
// instructions are bound by their issue, hence two issuers (4096 x 4096 over K = 256: 286 us
// with TN = 128, 252 with TN = 64, 217 with two issuers; over K = 128: 204, 178, 153; one row
// of tiles, K = 256: 49, 28, 26).
template <int TN_>
struct OzTile {
    static constexpr int TN = TN_, COLS = TN / 2;            // columns per epilogue warp
    // one producer, eight epilogue warps, and the issuers: for TN = 64 two, of a pass each
    static constexpr int ISSUERS = TN == 128 ? 1 : 2, NTHREADS = 32 * (9 + ISSUERS);
    static constexpr int STAGES = TN == 128 ? 3 : 4, STAGE = 192 * 1024 / STAGES;
    static constexpr int PLANE_B = TN * 32;                  // one digit of B in a stage
    static constexpr int NBUF = 512 / (2 * TN);              // accumulators: two weights of TN columns each
    // one weight's columns, and two weights' side by side
    static constexpr uint32_t IDESC1 =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
    static constexpr uint32_t IDESC2 = IDESC1 + ((uint32_t)(TN >> 3) << 17);
    // bytes of nd digits of both operands for a k16 step
    __device__ static constexpr uint32_t step_bytes(int nd) { return (uint32_t)nd * (PLANE + PLANE_B); }
};

// ---------------------------------------------------------------- digits
// Exponents of rows as stored beside the digits: the largest e + EXB of a row, e the biased
// exponent of a value after its scaling along k; 0 for a row of zeros.
constexpr int EXB = 8192, SPECIAL = 1 << 20;  // SPECIAL: the row holds an infinity or a NaN
// Scales along k: the largest (exponent of a value - largest of its column of B) + QB; 0: zeros
constexpr int QB = 4096;

// the biased exponent (1 for the subnormal numbers), 0 for zero, 0x7ff for an infinity or a NaN
__device__ __forceinline__ int exponent_of(double x) {
    const int hi = __double2hiint(x) & 0x7fffffff;
    return hi >= 1 << 20 ? hi >> 20 : (hi | __double2loint(x)) != 0;
}
// + the shift of its k (below 0: dropped); 0 stays zero
__device__ __forceinline__ int stored_exponent(double x, int shift) {
    const int e = exponent_of(x);
    return e == 0x7ff ? SPECIAL : e ? e + shift + EXB : 0;
}
// What the values at index k of an operand are shifted by: A (sign 1) down by as much as B
// (sign -1) up, so that the largest values of every row of B are about the same.  Where B's row is
// zero A's values do not matter, and DROP takes them below every other.
constexpr int DROP = -(1 << 16);
__device__ __forceinline__ int shift_at(const int* __restrict__ q, int k, int sign) {
    const int v = q ? q[k] : QB;
    return v ? sign * (v - QB) : sign > 0 ? DROP : 0;
}

// q[k] = the largest exponent of B's row k, each column taken relative to its own largest one (K
// <= FUSED_K: 32 columns per CTA, their exponents in shared memory; columns with an infinity
// or a NaN do not count).  Bound by the latency of its loads, hence eight in flight per thread:
// 256 k x 3840 columns 6 us, 20 with one.
constexpr int FUSED_K = 512, LOADS = 8;  // loads in flight per thread
__global__ void __launch_bounds__(256) oz_scale_fused(const double* __restrict__ b, long long rs, long long ks, int rows,
                                                      int k, int* __restrict__ q) {
    extern __shared__ int xe[];  // [k][33]
    __shared__ int em[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r0 = blockIdx.x * 32;
    if (threadIdx.x < 32) em[lane] = 0;
    __syncthreads();
    if (ks == 1) {
        for (int r = w; r < 32; r += 8) {
            int m = 0;
            for (int c0 = lane; c0 < k; c0 += 32 * LOADS) {
                double x[LOADS];
#pragma unroll
                for (int u = 0; u < LOADS; ++u) x[u] = r0 + r < rows && c0 + 32 * u < k ? b[(r0 + r) * rs + c0 + 32 * u] : 0.0;
#pragma unroll
                for (int u = 0; u < LOADS; ++u) {
                    const int e = exponent_of(x[u]);
                    if (c0 + 32 * u < k) xe[(c0 + 32 * u) * 33 + r] = e;
                    m = max(m, e);
                }
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) em[r] = m;
        }
    } else {
        int m = 0;
        for (int c0 = w; c0 < k; c0 += 8 * LOADS) {
            double x[LOADS];
#pragma unroll
            for (int u = 0; u < LOADS; ++u) x[u] = r0 + lane < rows && c0 + 8 * u < k ? b[r0 + lane + (c0 + 8 * u) * ks] : 0.0;
#pragma unroll
            for (int u = 0; u < LOADS; ++u) {
                const int e = exponent_of(x[u]);
                if (c0 + 8 * u < k) xe[(c0 + 8 * u) * 33 + lane] = e;
                m = max(m, e);
            }
        }
        if (m) atomicMax(em + lane, m);
    }
    __syncthreads();
    // a thread per k: its 32 columns
    for (int c = threadIdx.x; c < k; c += 256) {
        int m = 0;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
            const int e = xe[c * 33 + r], E = em[r];
            m = max(m, e && E != 0x7ff ? e - E + QB : 0);
        }
        if (m) atomicMax(q + c, m);
    }
}

// The same from the columns' exponents (unscaled, in ex): a thread per k and 32 columns where k is
// contiguous, a thread per column and 32 k where the columns are.
__global__ void __launch_bounds__(128) oz_scale(const double* __restrict__ b, long long rs, long long ks, int rows, int k,
                                                const int* __restrict__ ex, int* __restrict__ q) {
    if (ks == 1) {
        const int c = blockIdx.y * 128 + threadIdx.x, r1 = min(rows, (int)(blockIdx.x + 1) * 32);
        if (c >= k) return;
        int m = 0;
        for (int r0 = blockIdx.x * 32; r0 < r1; r0 += LOADS) {
            double x[LOADS];
#pragma unroll
            for (int u = 0; u < LOADS; ++u) x[u] = r0 + u < r1 ? b[(r0 + u) * rs + c] : 0.0;
#pragma unroll
            for (int u = 0; u < LOADS; ++u) {
                const int e = exponent_of(x[u]), E = r0 + u < r1 ? ex[r0 + u] : SPECIAL;
                m = max(m, e && E != SPECIAL ? e + EXB - E + QB : 0);
            }
        }
        if (m) atomicMax(q + c, m);
    } else {
        const int r = blockIdx.x * 128 + threadIdx.x, c1 = min(k, (int)(blockIdx.y + 1) * 32);
        const int E = r < rows ? ex[r] : SPECIAL;
#pragma unroll 4
        for (int c = blockIdx.y * 32; c < c1; ++c) {
            const int e = E != SPECIAL ? exponent_of(b[r * rs + c * ks]) : 0;
            const int m = __reduce_max_sync(0xffffffffu, e ? e + EXB - E + QB : 0);
            if ((threadIdx.x & 31) == 0 && m) atomicMax(q + c, m);
        }
    }
}

__global__ void oz_exponent_rows(const double* __restrict__ a, long long rs, long long ks, int rows, int k, int kper,
                                 int* __restrict__ ex, long long bs, int eb, const int* __restrict__ q, int sign) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const int c1 = min(k, (int)(blockIdx.y + 1) * kper);
    int m = 0;
    for (int c0 = blockIdx.y * kper; c0 < c1; c0 += LOADS) {
        double x[LOADS];
#pragma unroll
        for (int u = 0; u < LOADS; ++u) x[u] = c0 + u < c1 ? a[r * rs + (c0 + u) * ks] : 0.0;
#pragma unroll
        for (int u = 0; u < LOADS; ++u) m = max(m, stored_exponent(x[u], c0 + u < c1 ? shift_at(q, c0 + u, sign) : 0));
    }
    if (m) atomicMax(ex + r, m);
}

// contiguous along k: a warp per row
__global__ void oz_exponent_cols(const double* __restrict__ a, long long rs, int rows, int k, int* __restrict__ ex,
                                 long long bs, int eb, const int* __restrict__ q, int sign) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    int m = 0;
    for (int c0 = lane; c0 < k; c0 += 32 * LOADS) {
        double x[LOADS];
#pragma unroll
        for (int u = 0; u < LOADS; ++u) x[u] = c0 + 32 * u < k ? a[r * rs + c0 + 32 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < LOADS; ++u)
            m = max(m, stored_exponent(x[u], c0 + 32 * u < k ? shift_at(q, c0 + 32 * u, sign) : 0));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) ex[r] = m;
}

// x 2^shift as a 64-bit fixed-point number in units of 2^(E - EXB - 1085), E the row's stored
// exponent: |x 2^shift| < 2^(E - EXB - 1022), so the magnitude stays below 2^63.
__device__ __forceinline__ long long fixed64(double x, int shift, int E) {
    const long long b = __double_as_longlong(x);
    int e = (int)(b >> 52) & 0x7ff;
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    else e = 1;
    m <<= 10;
    const int sh = E - (e + shift + EXB);
    if (sh > 0) m = sh > 63 ? 0 : (m + (1ull << (sh - 1))) >> sh;
    return b < 0 ? -(long long)m : (long long)m;
}

// The digits of eight values of one row: 16 bytes of each of the eight planes.
__device__ __forceinline__ void store_digits(const double (&x)[8], const int (&shift)[8], int E, uint4* o, int digit) {
    uint32_t w[DIGITS][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        long long v = fixed64(x[j], shift[j], E);
#pragma unroll
        for (int s = DIGITS - 1; s >= 0; --s) {
            int d;
            if (s > 0) {
                d = (int)(signed char)(v & 0xff);
                v = (v - d) >> 8;
            } else {
                d = (int)v;
            }
            // the integer as FP32 (12582912 = 1.5 * 2^23), its upper half is the BF16
            const uint32_t f = __float_as_uint(__int_as_float(0x4b400000 + d) - 12582912.f);
            if (j & 1) w[s][j >> 1] |= f & 0xffff0000u;
            else w[s][j >> 1] = f >> 16;
        }
    }
#pragma unroll
    for (int s = 0; s < DIGITS; ++s) o[s * digit] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// Where the first digit of row r's half h of k16 step kb goes, in blocks of rb rows.
__device__ __forceinline__ long long digit_at(int r, int kb, int h, int k16, int rb) {
    const int i = r & (rb - 1);
    return ((long long)(rb == TILE ? r >> 7 : r >> 6) * k16 + kb) * (rb * 16) + (i >> 3) * 16 + h * 8 + (i & 7);
}

// Eight values along k of one row per thread -> 16 bytes of each digit plane.
// block.x = 128 rows, block.y = 2 halves of a k16 step; grid.x = row blocks,
// grid.y strides over the k16 steps.
__global__ void __launch_bounds__(256) oz_split(const double* __restrict__ a, long long rs, long long ks, int rows,
                                                int k, int k16, const int* __restrict__ ex, uint4* __restrict__ out,
                                                long long bs, int eb, int rb, const int* __restrict__ q, int sign) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    out += (long long)blockIdx.z * (eb / TILE) * k16 * (BLOCK / 16);
    const int r = blockIdx.x * TILE + threadIdx.x;
    const int E = r < rows ? ex[r] : 0;
    const bool ok = r < rows && E != SPECIAL;
    for (int kb = blockIdx.y; kb < k16; kb += gridDim.y) {
        const int c0 = kb * 16 + threadIdx.y * 8;
        double x[8];
        int sh[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const bool in = ok && c0 + j < k;
            x[j] = in ? a[r * rs + (c0 + j) * ks] : 0.0;
            sh[j] = in ? shift_at(q, c0 + j, sign) : 0;
        }
        store_digits(x, sh, E, out + digit_at(r, kb, threadIdx.y, k16, rb), rb * 2);
    }
}

// Exponents and digits in one launch for k <= FUSED_K (the panels of the factorisations
// and solves): a CTA holds 32 rows' values of all k in shared memory, so each is read
// from global memory once.  About 90 integer operations per value bound it: with 128
// rows per CTA a 3840 x 128 panel sat on 30 SMs for 20 us.
// blockIdx.y: one of two operands.  A and B of a product take one launch, in which the smaller
// one's CTAs run beside the other's (two launches: level 3 swimmer 21.50 ms, 20.98 with one;
// n = 700 with 64 right-hand sides 2.58 and 2.39), which pays for the scales' pass.
constexpr int FUSED_SMEM = FUSED_K * 33 * 8;
struct SplitOperand {
    const double* a;
    long long rs, ks, bs;
    int* ex;
    uint4* out;
    int rows, eb, rb, sign;
};
__global__ void __launch_bounds__(256) oz_split_fused(const __grid_constant__ SplitOperand s0,
                                                      const __grid_constant__ SplitOperand s1, int k, int k16,
                                                      const int* __restrict__ q) {
    const SplitOperand& S = blockIdx.y ? s1 : s0;
    const long long rs = S.rs, ks = S.ks;
    const int rows = S.rows, rb = S.rb, sign = S.sign;
    const double* __restrict__ a = S.a + blockIdx.z * S.bs;
    int* __restrict__ ex = S.ex + (long long)blockIdx.z * S.eb;
    uint4* __restrict__ out = S.out + (long long)blockIdx.z * (S.eb / TILE) * k16 * (BLOCK / 16);
    extern __shared__ double xs[];  // [k][33]
    __shared__ int em[32], sk[FUSED_K];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r0 = blockIdx.x * 32;
    if (r0 >= rows) return;
    const int kp = k16 * 16;
    if (threadIdx.x < 32) em[lane] = 0;
    for (int c = threadIdx.x; c < kp; c += 256) sk[c] = c < k ? shift_at(q, c, sign) : 0;
    __syncthreads();
    if (ks == 1) {
        for (int r = w; r < 32; r += 8) {
            int m = 0;
            for (int c0 = lane; c0 < kp; c0 += 32 * LOADS) {
                double x[LOADS];
#pragma unroll
                for (int u = 0; u < LOADS; ++u) x[u] = r0 + r < rows && c0 + 32 * u < k ? a[(r0 + r) * rs + c0 + 32 * u] : 0.0;
#pragma unroll
                for (int u = 0; u < LOADS; ++u) {
                    const int c = c0 + 32 * u;
                    if (c >= kp) break;
                    xs[c * 33 + r] = x[u];
                    m = max(m, stored_exponent(x[u], sk[c]));
                }
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) em[r] = m;
        }
    } else {
        int m = 0;
        for (int c0 = w; c0 < kp; c0 += 8 * LOADS) {
            double x[LOADS];
#pragma unroll
            for (int u = 0; u < LOADS; ++u) x[u] = r0 + lane < rows && c0 + 8 * u < k ? a[r0 + lane + (c0 + 8 * u) * ks] : 0.0;
#pragma unroll
            for (int u = 0; u < LOADS; ++u) {
                const int c = c0 + 8 * u;
                if (c >= kp) break;
                xs[c * 33 + lane] = x[u];
                m = max(m, stored_exponent(x[u], sk[c]));
            }
        }
        if (m) atomicMax(em + lane, m);
    }
    __syncthreads();
    const int E = em[lane];
    if (w == 0 && r0 + lane < rows) ex[r0 + lane] = E;
    for (int o8 = w; o8 < 2 * k16; o8 += 8) {
        double x[8];
        int sh[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = E != SPECIAL ? xs[(o8 * 8 + j) * 33 + lane] : 0.0;
            sh[j] = sk[o8 * 8 + j];
        }
        store_digits(x, sh, E, out + digit_at(r0 + lane, o8 >> 1, o8 & 1, k16, rb), rb * 2);
    }
}

// ---------------------------------------------------------------- product
struct OzArgs {
    const uint8_t *A, *B;     // digit blocks
    const int *exA, *exB;
    int M, N, K, k16;
    int tiles_m, tiles_n;
    double alpha, beta;
    double* C;
    long long ldc;
    const double *srcA, *srcB;  // rows with an infinity or a NaN are summed from these
    long long ars, aks, brs, bks;
    int batch;
    long long cb, abs, bbs;     // batch strides of C and of the sources
    long long* stash;           // 16384 sums per CTA
    int* err;
    long long wait;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"((unsigned long long)src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void red_add(double* p, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// K-major, no swizzle: 8-row core matrices of 128 bytes, the second half of the 16 k 128 bytes
// on (LBO), the next 8 rows 256 bytes on (SBO), so that half a block's rows are one piece;
// descriptor version 1.
__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
           (1ull << 46);
}

// C tiles in groups of 12 tile rows, the rows innermost: 152 CTAs then cover a patch
// of about 12 x 13 tiles, whose operands are re-read from L2 and not from HBM.
__device__ __forceinline__ void tile_at(const OzArgs& g, int t, int& b, int& tm, int& tn) {
    const int one = g.tiles_m * g.tiles_n;
    b = t / one;
    t -= b * one;
    const int per = 12 * g.tiles_n, grp = t / per, r = t - grp * per;
    const int h = min(12, g.tiles_m - grp * 12);
    tn = r / h;
    tm = grp * 12 + r - tn * h;
}

// What runs over the k16 steps [k0, k1) with nd digits of both operands in the stages: pass p
// (the weights 2p, 2p + 1), for SHORT also p + 1.  The long kernel has one pass
// between two read-outs: the leading passes 0, 1 alternate over HI_CHUNK steps, then 2 over
// MID_CHUNK and 3 over LO_CHUNK.  SHORT has accumulators for all four and loads a step's digits
// twice, not four times: four digits for passes 0 and 1, then all eight for 2 and 3.
struct Group {
    int p, nd, k0, k1;
    bool last_hi;
};
__device__ __forceinline__ int n_chunks(int k16, int chunk) { return (k16 + chunk - 1) / chunk; }
template <bool SHORT>
__device__ __forceinline__ int n_groups(int k16) {
    if (SHORT) return 2;
    return 2 * n_chunks(k16, HI_CHUNK) + n_chunks(k16, MID_CHUNK) + n_chunks(k16, LO_CHUNK);
}
template <bool SHORT>
__device__ __forceinline__ Group group_at(int q, int k16) {
    if (SHORT) return Group{2 * q, 4 * q + 4, 0, k16, false};
    const int nh = 2 * n_chunks(k16, HI_CHUNK), nm = n_chunks(k16, MID_CHUNK);
    const int p = q < nh ? q & 1 : q < nh + nm ? 2 : 3;
    const int c = q < nh ? HI_CHUNK : q < nh + nm ? MID_CHUNK : LO_CHUNK;
    const int k0 = (q < nh ? q >> 1 : q < nh + nm ? q - nh : q - nh - nm) * c;
    return Group{p, 2 * p + 2, k0, min(k16, k0 + c), q == nh - 1};
}

// The products of one k16 step of pass P.  Digit i of A goes with B's digits 2P - i and
// 2P - i + 1 in one instruction: these lie one behind the other in the stage, as the two
// weights' accumulators do in tensor memory, so the pair is one operand of 2 TN rows.  36
// instructions of TN columns per step issued at 93 clocks each, whatever TN; these 20 (16 of
// them of 2 TN) keep the tensor core busy and read A's digits from shared memory half as often.
template <int P, class T>
__device__ __forceinline__ void issue_step(uint32_t a0, uint32_t b0, uint32_t d, bool first) {
    constexpr int ND = 2 * P + 2;
    const uint64_t da = oz_desc(a0), db = oz_desc(b0);
    if (elect_one()) {
#pragma unroll
        for (int i = 0; i < ND - 1; ++i)
            mma_bf16(d, da + (uint64_t)(i * (PLANE >> 4)), db + (uint64_t)((ND - 2 - i) * (T::PLANE_B >> 4)), T::IDESC2,
                     first && i == 0 ? 0u : 1u);
        mma_bf16(d + T::TN, da + (uint64_t)((ND - 1) * (PLANE >> 4)), db, T::IDESC1, 1u);
    }
    __syncwarp();
}

// m 2^(e - 1075) where that is not a normal number (kept out of line: the read-out's code
// has to stay within the instruction cache).
__device__ __noinline__ double scale_far(unsigned long long m, int e) {
    return scalbn((double)m, max(-3000, min(3000, e - 1075)));
}

// (hi 2^32 + lo) 2^(56 + Ea + Eb - 2170) to nearest even, in integer arithmetic (an FP64
// operation per element costs a tile 5 us)
__device__ __forceinline__ double round96(long long hi, long long lo, int Eab) {
    long long h = hi + (lo >> 32);
    uint32_t l = (uint32_t)lo;
    const uint32_t neg = (uint32_t)(h >> 63);
    if (neg) {
        h = ~h + (l == 0);
        l = 0u - l;
    }
    if (h == 0 && l == 0) return 0.0;
    // shift the 96 bits left until the top bit is set
    int lz = 0;
    if (h == 0) {
        h = (long long)((unsigned long long)l << 32);
        l = 0;
        lz = 64;
    }
    const int z = __clzll(h);
    lz += z;
    const unsigned long long L = (unsigned long long)l << 32;
    const unsigned long long T = ((unsigned long long)h << z) | ((L >> 1) >> (63 - z));
    unsigned long long m = T >> 11;
    const uint32_t rb = (uint32_t)T & 0x7ff, sticky = (uint32_t)((L << z) != 0) | (uint32_t)(m & 1);
    m += rb + (sticky ? 1 : 0) > 0x400 ? 1 : 0;
    const int e = Eab - lz - 996;
    double r;
    if (e > 0 && e < 2046) r = __longlong_as_double((long long)(((unsigned long long)(e - 1) << 52) + m));
    else r = scale_far(m, e);
    return __hiloint2double(__double2hiint(r) ^ (int)(neg & 0x80000000u), __double2loint(r));
}

// s 2^16 + q, |q| < 2^35, as hi 2^32 + lo.
__device__ __forceinline__ void parts80(long long s, long long q, long long& hi, uint32_t& lo) {
    const long long x = (long long)((unsigned long long)(uint32_t)s << 16) + q;
    lo = (uint32_t)x;
    hi = ((long long)(int)(s >> 32) << 16) + (int)(x >> 32);
}
__device__ __noinline__ double round80_far(long long s, float v0, float v1, int Eab) {
    long long hi;
    uint32_t lo;
    parts80(s, (long long)__float2int_rn(v0) * 256 + __float2int_rn(v1), hi, lo);
    return round96(hi, lo, Eab);
}
// (s 2^16 + v0 2^8 + v1) 2^(56 + Ea + Eb - 2170) to nearest even for eight elements: integer
// arithmetic (two FP64 operations per element took a 128 x 128 tile 9 us), branch-free but for
// one rare test of all eight (a branch per element kept their latencies from overlapping, 750
// cycles each).
__device__ __forceinline__ void round80(const long long* s, const float (&v0)[8], const float (&v1)[8],
                                        const int (&E)[8], double (&r)[8]) {
    uint32_t far = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        long long h;
        uint32_t l;
        parts80(s[j], (long long)__float2int_rn(v0[j]) * 256 + __float2int_rn(v1[j]), h, l);
        const uint32_t neg = (uint32_t)((int)(h >> 32) >> 31);
        const unsigned long long a =
            ((unsigned long long)h ^ ((unsigned long long)neg << 32 | neg)) + ((neg & 1) & (uint32_t)(l == 0));
        l = (l ^ neg) - neg;
        const int z = __clzll((long long)a) & 63;
        const unsigned long long L = (unsigned long long)l << 32;
        const unsigned long long T = (a << z) | ((L >> 1) >> (63 - z));
        unsigned long long m = T >> 11;
        const uint32_t rb = (uint32_t)T & 0x7ff, sticky = (uint32_t)((L << z) != 0) | (uint32_t)(m & 1);
        m += rb + sticky > 0x400 ? 1 : 0;
        const int e = E[j] - z - 996;
        far |= (uint32_t)(e - 1) >= 2045u || a == 0 ? 1u << j : 0u;
        m += (unsigned long long)(uint32_t)(e - 1) << 52;
        r[j] = __hiloint2double((int)(m >> 32) ^ (int)(neg & 0x80000000u), (int)m);
    }
    if (far) {
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
            if (!(far >> j & 1)) continue;
            long long x = s[0];
            float f0 = v0[0], f1 = v1[0];
            int Ej = E[0];
#pragma unroll
            for (int u = 1; u < 8; ++u) {
                x = j == u ? s[u] : x;
                f0 = j == u ? v0[u] : f0;
                f1 = j == u ? v1[u] : f1;
                Ej = j == u ? E[u] : Ej;
            }
            const double f = round80_far(x, f0, f1, Ej);
#pragma unroll
            for (int u = 0; u < 8; ++u) r[u] = j == u ? f : r[u];
        }
    }
}

// SHORT: k16 <= HI_CHUNK
template <bool SHORT, class T>
__global__ void __launch_bounds__(T::NTHREADS, 1) oz_gemm_kernel(const __grid_constant__ OzArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int STAGES = T::STAGES, STAGE = T::STAGE, TN = T::TN, COLS = T::COLS, NBUF = T::NBUF;
    static_assert(!SHORT || (NBUF == 4 && T::ISSUERS == 2), "SHORT has an accumulator and, of two, an issuer per pass");
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * STAGES), tempty0 = smem_u32(bars + 2 * STAGES + NBUF);
    const uint32_t done_bar = smem_u32(bars + 2 * STAGES + 2 * NBUF);
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 2 * NBUF + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int tiles = g.tiles_m * g.tiles_n * g.batch, k16 = g.k16, ng = n_groups<SHORT>(k16);
    const bool halves = SHORT && k16 > MID_CHUNK;  // pass 2 read out after mid steps too
    const int mid = (k16 + 1) / 2;
    static_assert(!SHORT || (HI_CHUNK + 1) / 2 <= MID_CHUNK, "two halves suffice");
    static_assert(!SHORT || T::step_bytes(DIGITS) == STAGE, "a stage per step in passes 2 and 3: mid starts one");
    int* const err = g.err;
    const long long wait = g.wait;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, T::ISSUERS);
        }
        for (int a = 0; a < NBUF; ++a) {
            mbar_init(tfull0 + 8 * a, 1);
            mbar_init(tempty0 + 8 * a, 256);
        }
        mbar_init(done_bar, T::ISSUERS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---------------- producer
        int s = 0;
        uint32_t ph = 0;
        int armed[STAGES] = {};
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            int tb, tm, tn;
            tile_at(g, t, tb, tm, tn);
            const uint8_t* A = g.A + ((long long)tb * g.tiles_m + tm) * k16 * BLOCK;
            const long long bn = TN == TILE ? (long long)tb * g.tiles_n + tn : (long long)tb * ((g.tiles_n + 1) & ~1) + tn;
            const uint8_t* B = g.B + bn * k16 * (DIGITS * T::PLANE_B);
            for (int q = 0; ok && q < ng; ++q) {
                const Group G = group_at<SHORT>(q, k16);
                const int nd = G.nd, step = T::step_bytes(nd), sp = STAGE / step;
                for (int k = G.k0; k < G.k1; k += sp) {
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1, err, wait)) { ok = false; break; }
                    const int n = min(sp, G.k1 - k);
                    uint32_t dst = smem_u32(smem + s * STAGE);
                    const uint32_t fb = full0 + 8 * s;
                    mbar_expect_tx(fb, step * n);
                    for (int u = 0; u < n; ++u) {
                        bulk_load(dst, A + (long long)(k + u) * BLOCK, nd * PLANE, fb);
                        bulk_load(dst + nd * PLANE, B + (long long)(k + u) * (DIGITS * T::PLANE_B), nd * T::PLANE_B, fb);
                        dst += step;
                    }
                    armed[s] += 1;
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
        // drain: every armed stage must have completed before the CTA exits
        for (int q = 0; q < STAGES; ++q)
            if (armed[q] > 0) {
                const uint32_t par = (uint32_t)((armed[q] - 1) & 1);
                const long long t0 = clock64();
                while (!mbar_try(full0 + 8 * q, par) && clock64() - t0 < DRAIN_CYCLES) {
                }
            }
    } else if (warp == 1 || warp >= 10) {
        // ---------------- MMA issuer (of pass `mine` of a group): the whole warp runs the
        // loop, so that the descriptors are uniform values, and one lane issues
        const int mine = warp == 1 ? 0 : 1;
        int s = 0, acc = 0;
        uint32_t ph = 0, aph = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            for (int q = 0; ok && q < ng; ++q) {
                const Group G = group_at<SHORT>(q, k16);
                const int step = T::step_bytes(G.nd), sp = STAGE / step;
                const int p = G.p + mine;
                if (SHORT) acc = p;
                // SHORT: pass 2's accumulator is used twice per tile, with the parities 0 and 1
                const bool two = halves && p == 2;
                ok = __all_sync(0xffffffffu, mbar_wait(tempty0 + 8 * acc, two ? 1u : aph ^ 1, err, wait));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(acc * 2 * TN);
                for (int k = G.k0; k < G.k1; k += sp) {
                    if (two && k == mid) {
                        if (elect_one()) mma_commit(tfull0 + 8 * acc);
                        __syncwarp();
                        ok = __all_sync(0xffffffffu, mbar_wait(tempty0 + 8 * acc, 0, err, wait));
                        if (!ok) break;
                        tc_fence_after();
                    }
                    ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, ph, err, wait));
                    if (!ok) break;
                    tc_fence_after();
                    const int n = min(sp, G.k1 - k);
                    uint32_t a0 = smem_u32(smem + s * STAGE);
                    for (int u = 0; u < n; ++u, a0 += step) {
                        const bool first = k + u == G.k0 || (two && k + u == mid);
                        const uint32_t b0 = a0 + G.nd * PLANE;
                        if (p == 0) issue_step<0, T>(a0, b0, d, first);
                        else if (p == 1) issue_step<1, T>(a0, b0, d, first);
                        else if (p == 2) issue_step<2, T>(a0, b0, d, first);
                        else issue_step<3, T>(a0, b0, d, first);
                    }
                    if (elect_one()) mma_commit(empty0 + 8 * s);
                    __syncwarp();
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                if (elect_one()) mma_commit(tfull0 + 8 * acc);
                __syncwarp();
                if (!SHORT && ++acc == NBUF) { acc = 0; aph ^= 1; }
            }
            if (SHORT) aph ^= 1;
        }
        // all MMAs issued by this CTA complete before TMEM is released
        if (elect_one()) mma_commit(done_bar);
        __syncwarp();
        const long long t0 = clock64();
        while (!mbar_try(done_bar, 0) && clock64() - t0 < DRAIN_CYCLES) {
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: row = TMEM lane, COLS columns per thread
        const int quarter = warp & 3, row = quarter * 32 + lane, col0 = ((warp - 2) >> 2) * COLS;
        long long* const stash = SHORT ? nullptr : g.stash + (long long)blockIdx.x * (TILE * TILE) + col0 * TILE + row;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        int acc = 0;
        uint32_t aph = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            int tb, tm, tn;
            tile_at(g, t, tb, tm, tn);
            const int* const exA = g.exA + (long long)tb * g.tiles_m * TILE;
            const int* const exB = g.exB + (long long)tb * ((g.N + TILE - 1) / TILE) * TILE;
            const int m = tm * TILE + row, n0 = tn * TN + col0, nc = min(COLS, g.N - n0);
            const bool mine = m < g.M;
            // exponents: this thread's row, and one or two of the warp's columns per lane
            const int Ea = mine ? exA[m] : 0;
            const int Eb0 = lane < nc ? exB[n0 + lane] : 0, Eb1 = COLS > 32 && lane + 32 < nc ? exB[n0 + 32 + lane] : 0;
            const bool special = __any_sync(0xffffffffu, Ea == SPECIAL || Eb0 == SPECIAL || Eb1 == SPECIAL);
            const int ea = Ea - 2 * EXB;
            double* const Cm = g.C + tb * g.cb + m + (long long)n0 * g.ldc;
            const double alpha = g.alpha, beta = g.beta;
            long long sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0;
            // The read-out walks the columns eight at a time in a rolled loop, the sums moving
            // down by eight registers each turn: unrolled it outgrew the instruction cache and
            // took 70 us a tile.
            // C += v goes to L2 as a reduction (one per element, IEEE rounding): reading C
            // here left the warps waiting on its loads for two thirds of the read-out.
            const int flip = alpha == -1.0 ? 0x80000000 : 0;
            // Elements whose row or column holds an infinity or a NaN (zero digits) are left out here
            // and follow below.
            const bool plain = (alpha == 1.0 || alpha == -1.0) && (beta == 0.0 || beta == 1.0) && !special,
                       add = beta == 1.0;
            const uint32_t skip0 = __ballot_sync(0xffffffffu, Eb0 == SPECIAL), skip1 = __ballot_sync(0xffffffffu, Eb1 == SPECIAL);
            auto left_out = [&](int c) { return Ea == SPECIAL || ((COLS <= 32 || c < 32 ? skip0 : skip1) >> (c & 31) & 1); };
            auto finish = [&](int c, const double (&r)[8]) {
                if (plain && add) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (mine && c + j < nc)
                            red_add(Cm + (long long)(c + j) * g.ldc,
                                    __hiloint2double(__double2hiint(r[j]) ^ flip, __double2loint(r[j])));
                } else if (plain) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (mine && c + j < nc)
                            Cm[(long long)(c + j) * g.ldc] =
                                __hiloint2double(__double2hiint(r[j]) ^ flip, __double2loint(r[j]));
                } else {
#pragma unroll 1
                    for (int j = 0; j < 8; ++j) {
                        if (!mine || c + j >= nc) break;
                        if (special && left_out(c + j)) continue;
                        double* const p = Cm + (long long)(c + j) * g.ldc;
                        double v = r[0];
#pragma unroll
                        for (int u = 1; u < 8; ++u) v = j == u ? r[u] : v;
                        *p = beta == 0.0 ? alpha * v : fma(alpha, v, beta * *p);
                    }
                }
            };
            auto exps = [&](int c) { return ea + __shfl_sync(0xffffffffu, COLS <= 32 || c < 32 ? Eb0 : Eb1, c & 31); };
            auto rotate = [&]() {
#pragma unroll
                for (int j = 0; j < COLS - 8; ++j) sum[j] = sum[j + 8];
            };
            for (int q = 0; q < (SHORT ? NBUF + halves : ng); ++q) {
                const int p = SHORT ? q - (halves && q > 2) : group_at<SHORT>(q, k16).p;
                uint32_t par = aph;
                if (SHORT) {
                    acc = p;
                    if (halves && p == 2) par = q - 2;
                }
                // the whole warp stays or leaves: tcgen05.ld is warp-collective
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, par, err, wait));
                if (!ok) break;
                tc_fence_after();
                const uint32_t base = tmem_base + lanes + (uint32_t)(acc * 2 * TN + col0);
                if (SHORT && p == 3) {
#pragma unroll 1
                    for (int c = 0; c < COLS; c += 8) {
                        float v0[8], v1[8];
                        tmem_ld8x2(base + c, base + TN + c, v0, v1);
                        double r[8];
                        int E[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) E[j] = exps(c + j);
                        round80(sum, v0, v1, E, r);
                        finish(c, r);
                        rotate();
                    }
                } else {
                    // weights of the two accumulators within the sums (SHORT: of 0 to 5 in units
                    // of weight 5, below 2^63)
                    const long long w1 = SHORT ? 1ll << (32 - 16 * p) : p & 1 ? 1 : 1 << 16;
                    const long long w0 = w1 << 8;
#pragma unroll
                    for (int c = 0; c < COLS; c += 16) {
                        float v[16];
                        tmem_ld16(base + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[c + j] += (long long)__float2int_rn(v[j]) * w0;
                        tmem_ld16(base + TN + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[c + j] += (long long)__float2int_rn(v[j]) * w1;
                    }
                }
                tc_fence_before();
                mbar_arrive(tempty0 + 8 * acc);
                if (!SHORT && ++acc == NBUF) { acc = 0; aph ^= 1; }
                if (!SHORT && group_at<SHORT>(q, k16).last_hi) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j) {
                        stash[j * TILE] = sum[j];
                        sum[j] = 0;
                    }
                }
            }
            if (!ok) break;
            if (SHORT) aph ^= 1;
            if (!SHORT) {
#pragma unroll 1
                for (int c = 0; c < COLS; c += 8) {
                    double r[8];
                    long long h[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) h[j] = stash[(c + j) * TILE];
#pragma unroll
                    for (int j = 0; j < 8; ++j) r[j] = round96(h[j], sum[j], exps(c + j));
                    finish(c, r);
                    rotate();
                }
            }
            if (special && mine) {
                // plain sums, or NaN where C takes the place of B
                for (int c = 0; c < nc; ++c) {
                    if (!left_out(c)) continue;
                    const long long n = n0 + c;
                    double r = g.srcB ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
                    for (int k = 0; g.srcB && k < g.K; ++k)
                        r = fma(g.srcA[tb * g.abs + m * g.ars + k * g.aks], g.srcB[tb * g.bbs + n * g.brs + k * g.bks], r);
                    double* const o = Cm + c * g.ldc;
                    *o = beta == 0.0 ? alpha * r : fma(alpha, r, beta * *o);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}

int g_sms = 0;
std::once_flag g_once;

}  // namespace

static void set_up() {
    std::call_once(g_once, [] {
        int dev = 0;
        CUDA_CHECK(cudaGetDevice(&dev));
        CUDA_CHECK(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
        CUDA_CHECK(cudaFuncSetAttribute(oz_gemm_kernel<true, OzTile<64>>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        SMEM_BYTES));
        CUDA_CHECK(cudaFuncSetAttribute(oz_gemm_kernel<false, OzTile<128>>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        SMEM_BYTES));
        CUDA_CHECK(cudaFuncSetAttribute(oz_scale_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_K * 33 * 4));
        CUDA_CHECK(cudaFuncSetAttribute(oz_split_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM));
    });
}

void OzMat::lay_out(const double* a, long long rs_, long long ks_, int rows_, int k_, cudaStream_t st, bool right_,
                    int batch_, long long bs_) {
    set_up();
    rows = rows_;
    k = k_;
    k16 = ceil_div(k, 16);
    batch = batch_;
    src = a;
    rs = rs_;
    ks = ks_;
    bs = bs_;
    right = right_;
    block = right && k16 <= HI_CHUNK ? 64 : TILE;
    const int nb = ceil_div(rows, TILE);
    d.alloc((size_t)batch * nb * k16 * (BLOCK / 16), st);
    ex.alloc((size_t)batch * nb * TILE, st);
}

// whether exponents and digits take one launch
static bool fused(const OzMat& m) { return m.k <= FUSED_K && (m.rs == 1 || m.ks == 1); }
static SplitOperand operand(const OzMat& m) {
    return {m.src, m.rs, m.ks, m.bs, m.ex.get(), m.d.get(), m.rows, ceil_div(m.rows, TILE) * TILE, m.block, m.right ? -1 : 1};
}

void OzMat::split(const double* a, long long rs_, long long ks_, int rows_, int k_, cudaStream_t st, bool right_,
                  int batch_, long long bs_, const int* q) {
    lay_out(a, rs_, ks_, rows_, k_, st, right_, batch_, bs_);
    split_values(q, st);
}

void OzMat::split_values(const int* q, cudaStream_t st) {
    const int sign = right ? -1 : 1;
    const int nb = ceil_div(rows, TILE), eb = nb * TILE;
    if (fused(*this)) {
        const SplitOperand s = operand(*this);
        LAUNCH(oz_split_fused, dim3(ceil_div(rows, 32), 1, batch), 256, k16 * 16 * 33 * 8, st, s, s, k, k16, q);
        return;
    }
    if (ks == 1) {
        LAUNCH(oz_exponent_cols, dim3(ceil_div(rows, 8), 1, batch), 256, 0, st, src, rs, rows, k, ex.get(), bs, eb, q,
               sign);
    } else {
        ex.zero();
        const int kper = 32;
        LAUNCH(oz_exponent_rows, dim3(nb, ceil_div(k, kper), batch), TILE, 0, st, src, rs, ks, rows, k, kper, ex.get(),
               bs, eb, q, sign);
    }
    // about four CTAs per SM's worth of k16 steps
    const int gy = std::max(1, std::min(k16, 152 * 8 / (nb * batch)));
    LAUNCH(oz_split, dim3(nb, gy, batch), dim3(TILE, 2), 0, st, src, rs, ks, rows, k, k16, ex.get(), d.get(), bs,
           eb, block, q, sign);
}

void oz_gemm(const OzMat& A, const OzMat& B, double alpha, double beta, double* C, long long ldc, int* err,
             cudaStream_t st, long long cb) {
    if (A.rows <= 0 || B.rows <= 0 || A.batch <= 0) return;
    if (A.k != B.k || A.k <= 0 || A.batch != B.batch || ldc < A.rows || !err) fail(SQBEM_ERR_ARG, "oz_gemm: bad arguments");
    set_up();
    OzArgs g;
    g.A = reinterpret_cast<const uint8_t*>(A.d.get());
    g.B = reinterpret_cast<const uint8_t*>(B.d.get());
    g.exA = A.ex.get();
    g.exB = B.ex.get();
    g.M = A.rows;
    g.N = B.rows;
    g.K = A.k;
    g.k16 = A.k16;
    g.tiles_m = ceil_div(g.M, TILE);
    const bool brief = g.k16 <= HI_CHUNK;
    if (A.block != TILE || B.block != (brief ? 64 : TILE)) fail(SQBEM_ERR_ARG, "oz_gemm: B was not split as the right operand");
    g.tiles_n = ceil_div(g.N, B.block);
    g.alpha = alpha;
    g.beta = beta;
    g.C = C;
    g.ldc = ldc;
    g.srcA = A.src;
    g.ars = A.rs;
    g.aks = A.ks;
    g.srcB = C == B.src || C == A.src ? nullptr : B.src;
    g.brs = B.rs;
    g.bks = B.ks;
    g.batch = A.batch;
    g.cb = cb;
    g.abs = A.bs;
    g.bbs = B.bs;
    const int grid = std::min(g.tiles_m * g.tiles_n * g.batch, g_sms);
    DevBuf<long long> stash(brief ? 0 : (size_t)grid * TILE * TILE, st);
    g.stash = stash.get();
    g.err = err;
    g.wait = gemm_wait_cycles();
    // credited as BF16 tensor work: 36 digit products
    const double fl = 72.0 * g.batch * g.M * g.N * g.K,
                 by = g.batch * (16.0 * ((double)g.M + g.N) * g.K + (beta == 0.0 ? 8.0 : 16.0) * g.M * g.N);
    if (brief)
        TIMED_LAUNCH("oz_gemm", fl, by, (oz_gemm_kernel<true, OzTile<64>>), grid, OzTile<64>::NTHREADS, SMEM_BYTES, st, g);
    else
        TIMED_LAUNCH("oz_gemm", fl, by, (oz_gemm_kernel<false, OzTile<128>>), grid, OzTile<128>::NTHREADS, SMEM_BYTES, st, g);
}

void oz_scales(const double* B, long long rs, long long ks, int N, int K, int* q, cudaStream_t st) {
    set_up();
    if (K <= FUSED_K && (rs == 1 || ks == 1)) {
        LAUNCH(oz_scale_fused, ceil_div(N, 32), 256, K * 33 * 4, st, B, rs, ks, N, K, q);
        return;
    }
    DevBuf<int> ex(N, st);
    if (ks == 1) {
        LAUNCH(oz_exponent_cols, ceil_div(N, 8), 256, 0, st, B, rs, N, K, ex.get(), 0, 0, nullptr, 0);
        LAUNCH(oz_scale, dim3(ceil_div(N, 32), ceil_div(K, 128)), 128, 0, st, B, rs, ks, N, K, ex.get(), q);
    } else {
        ex.zero();
        LAUNCH(oz_exponent_rows, dim3(ceil_div(N, TILE), ceil_div(K, 32)), TILE, 0, st, B, rs, ks, N, K, 32, ex.get(), 0,
               0, nullptr, 0);
        LAUNCH(oz_scale, dim3(ceil_div(N, 128), ceil_div(K, 32)), 128, 0, st, B, rs, ks, N, K, ex.get(), q);
    }
}

void oz_product(const double* A, long long ars, long long aks, const double* B, long long brs, long long bks, int M, int N,
                int K, double alpha, double beta, double* C, long long ldc, int* err, cudaStream_t st, int* q) {
    DevBuf<int> own;
    if (!q) {
        own.alloc(K, st);
        own.zero();
        q = own.get();
    }
    oz_scales(B, brs, bks, N, K, q, st);
    OzMat a, b;
    a.lay_out(A, ars, aks, M, K, st, false);
    b.lay_out(B, brs, bks, N, K, st, true);
    if (fused(a) && fused(b)) {
        LAUNCH(oz_split_fused, dim3(ceil_div(std::max(M, N), 32), 2), 256, a.k16 * 16 * 33 * 8, st, operand(a), operand(b), K,
               a.k16, q);
    } else {
        a.split_values(q, st);
        b.split_values(q, st);
    }
    oz_gemm(a, b, alpha, beta, C, ldc, err, st);
}

}  // namespace sqbem
