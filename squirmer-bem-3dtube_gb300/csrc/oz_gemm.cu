// oz_gemm.cu -- the kernels of oz_gemm.cuh.
//
// GB300 multiplies FP64 at about 1 TFLOP/s and BF16 on the tensor cores at
// about 1900, so the 36 digit products of an FP64 product still leave room for a
// factor of forty.
//
// Tile 128 x 128 of C per CTA, one persistent CTA per SM:
//   warp 0     producer: bulk copies of the digits' blocks into a 3-stage ring of
//              64 KB stages (the blocks are stored in the order the MMA reads, so
//              the digits a pass needs of one k16 step are one copy per operand);
//   warp 1     MMA issuer: passes of two weights (d, d + 1) into the two halves of a
//              256-column accumulator, double-buffered over the 512 TMEM columns;
//   warps 2-9  epilogue: the accumulators as integers into 64-bit sums held in
//              registers (64 per thread), the rounding to FP64, C.
// Four passes: weights 0, 1 (digits 0-1) and 2, 3 (digits 0-3) in chunks of 256 k,
// where every sum is exact (4 * 256 * 2^14 = 2^24); then weights 4, 5 and 6, 7
// in chunks of 1024 k, whose rounding past 2^24 lies 2^-56 below the product
// of the largest entries.
//   K <= 256 (the panels' updates): the 64-bit sums also take weights 4 and 5 (2^62 at
//   most), and the last pass goes straight into the rounding.
//   K > 256: the sums of the leading passes wait in global scratch (L2) for the others,
//   since both sets do not fit in the registers together.
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
constexpr int STAGES = 3, STAGE = 64 * 1024;
// past the ring: room for the descriptors' strides, never read
constexpr int SMEM_BYTES = STAGES * STAGE + 1024 + 256;
constexpr int NTHREADS = 320;              // producer, issuer, 8 epilogue warps
constexpr int HI_CHUNK = 16, LO_CHUNK = 64;  // k16 steps between read-outs
constexpr uint32_t IDESC =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);

// ---------------------------------------------------------------- digits
__global__ void oz_exponent_rows(const double* __restrict__ a, long long rs, long long ks, int rows, int k, int kper,
                                 int* __restrict__ ex, long long bs, int eb) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const int c1 = min(k, (int)(blockIdx.y + 1) * kper);
    int m = 0;
#pragma unroll 8
    for (int c = blockIdx.y * kper; c < c1; ++c) m = max(m, __double2hiint(a[r * rs + c * ks]) & 0x7ff00000);
    if (m) atomicMax(ex + r, m >> 20);
}

// contiguous along k: a warp per row
__global__ void oz_exponent_cols(const double* __restrict__ a, long long rs, int rows, int k, int* __restrict__ ex,
                                 long long bs, int eb) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    int m = 0;
#pragma unroll 4
    for (int c = lane; c < k; c += 32) m = max(m, __double2hiint(a[r * rs + c]) & 0x7ff00000);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) ex[r] = m >> 20;
}

// x as a 64-bit fixed-point number in units of 2^(E - 1085), E the row's largest
// biased exponent: |x| < 2^(E - 1022), so the magnitude stays below 2^63.
__device__ __forceinline__ long long fixed64(double x, int E) {
    const long long b = __double_as_longlong(x);
    int e = (int)(b >> 52) & 0x7ff;
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    else e = 1;
    m <<= 10;
    const int sh = max(E, 1) - e;
    if (sh > 0) m = sh > 63 ? 0 : (m + (1ull << (sh - 1))) >> sh;
    return b < 0 ? -(long long)m : (long long)m;
}

// The digits of eight values of one row: 16 bytes of each of the eight planes.
__device__ __forceinline__ void store_digits(const double (&x)[8], int E, uint4* o) {
    uint32_t w[DIGITS][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        long long v = fixed64(x[j], E);
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
    for (int s = 0; s < DIGITS; ++s) o[s * (PLANE / 16)] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// Eight values along k of one row per thread -> 16 bytes of each digit plane.
// block.x = 128 rows, block.y = 2 halves of a k16 step; grid.x = row blocks,
// grid.y strides over the k16 steps.
__global__ void __launch_bounds__(256) oz_split(const double* __restrict__ a, long long rs, long long ks, int rows,
                                                int k, int k16, const int* __restrict__ ex, uint4* __restrict__ out,
                                                long long bs, int eb) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    out += (long long)blockIdx.z * (eb / TILE) * k16 * (BLOCK / 16);
    const int r = blockIdx.x * TILE + threadIdx.x;
    const int E = r < rows ? ex[r] : 0;
    const bool ok = r < rows && E != 0x7ff;
    for (int kb = blockIdx.y; kb < k16; kb += gridDim.y) {
        const int c0 = kb * 16 + threadIdx.y * 8;
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = ok && c0 + j < k ? a[r * rs + (c0 + j) * ks] : 0.0;
        store_digits(x, E, out + ((long long)blockIdx.x * k16 + kb) * (BLOCK / 16) + threadIdx.y * (PLANE / 32) + threadIdx.x);
    }
}

// Exponents and digits in one launch for k <= FUSED_K (the panels of the factorisations
// and solves): a CTA holds 32 rows' values of all k in shared memory, so each is read
// from global memory once.  About 90 integer operations per value bound it: with 128
// rows per CTA a 3840 x 128 panel sat on 30 SMs for 20 us.
constexpr int FUSED_K = 512;
constexpr int FUSED_SMEM = FUSED_K * 33 * 8;
__global__ void __launch_bounds__(256) oz_split_fused(const double* __restrict__ a, long long rs, long long ks, int rows,
                                                      int k, int k16, int* __restrict__ ex, uint4* __restrict__ out,
                                                      long long bs, int eb) {
    a += blockIdx.z * bs;
    ex += (long long)blockIdx.z * eb;
    out += (long long)blockIdx.z * (eb / TILE) * k16 * (BLOCK / 16);
    extern __shared__ double xs[];  // [k][33]
    __shared__ int em[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r0 = blockIdx.x * 32;
    if (threadIdx.x < 32) em[lane] = 0;
    __syncthreads();
    const int kp = k16 * 16;
    if (ks == 1) {
        for (int r = w; r < 32; r += 8) {
            int m = 0;
            for (int c = lane; c < kp; c += 32) {
                const double x = r0 + r < rows && c < k ? a[(r0 + r) * rs + c] : 0.0;
                xs[c * 33 + r] = x;
                m = max(m, __double2hiint(x) & 0x7ff00000);
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) em[r] = m >> 20;
        }
    } else {
        int m = 0;
        for (int c = w; c < kp; c += 8) {
            const double x = r0 + lane < rows && c < k ? a[r0 + lane + c * ks] : 0.0;
            xs[c * 33 + lane] = x;
            m = max(m, __double2hiint(x) & 0x7ff00000);
        }
        if (m) atomicMax(em + lane, m >> 20);
    }
    __syncthreads();
    const int E = em[lane];
    if (w == 0 && r0 + lane < rows) ex[r0 + lane] = E;
    uint4* const o = out + (long long)(blockIdx.x >> 2) * k16 * (BLOCK / 16) + (blockIdx.x & 3) * 32 + lane;
    for (int o8 = w; o8 < 2 * k16; o8 += 8) {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = E != 0x7ff ? xs[(o8 * 8 + j) * 33 + lane] : 0.0;
        store_digits(x, E, o + (o8 >> 1) * (BLOCK / 16) + (o8 & 1) * (PLANE / 32));
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

// K-major, no swizzle: 8-row core matrices of 128 bytes, the next 8 rows 128 bytes
// on (SBO), the second half of the 16 k 2048 bytes on (LBO); descriptor version 1.
__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(2048 >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
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

// One accumulation between two read-outs: pass p (weights 2p, 2p + 1) over the k16
// steps [k0, k1).  The leading passes 0, 1 alternate over HI_CHUNK steps, then 2, 3
// over LO_CHUNK.
struct Group {
    int p, k0, k1;
    bool last_hi, last;
};
__device__ __forceinline__ int n_groups(int k16) {
    return 2 * ((k16 + HI_CHUNK - 1) / HI_CHUNK) + 2 * ((k16 + LO_CHUNK - 1) / LO_CHUNK);
}
__device__ __forceinline__ Group group_at(int q, int k16) {
    const int nh = 2 * ((k16 + HI_CHUNK - 1) / HI_CHUNK), nl = 2 * ((k16 + LO_CHUNK - 1) / LO_CHUNK);
    Group g;
    const bool hi = q < nh;
    const int c = hi ? HI_CHUNK : LO_CHUNK, i = hi ? q : q - nh;
    g.p = (hi ? 0 : 2) + (i & 1);
    g.k0 = (i >> 1) * c;
    g.k1 = min(k16, g.k0 + c);
    g.last_hi = q == nh - 1;
    g.last = q == nh + nl - 1;
    return g;
}
// k16 steps per stage of pass p (2, 4, 6, 8 digits of both operands)
__device__ __forceinline__ int steps_per_stage(int p) { return p == 0 ? 4 : p == 1 ? 2 : 1; }

template <int P>
__device__ __forceinline__ void issue_step(uint32_t a0, uint32_t d, bool first) {
    constexpr int ND = 2 * P + 2;
    const uint64_t da = oz_desc(a0), db = oz_desc(a0 + ND * PLANE);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        constexpr int D0 = 2 * P;
#pragma unroll
        for (int i = 0; i <= D0 + h; ++i) {
            const int j = D0 + h - i;
            mma_bf16(d + h * TILE, da + (uint64_t)(i * (PLANE >> 4)), db + (uint64_t)(j * (PLANE >> 4)), IDESC,
                     first && i == 0 ? 0u : 1u);
        }
    }
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

// (s 2^16 + q) 2^(56 + Ea + Eb - 2170) to nearest even, |q| < 2^35: the high 32 bits and the
// low 48 each put into the significand of a power of two, whose removal and sum are two
// FP64 operations, the first exact.
__device__ __forceinline__ double significand80(long long s, long long q) {
    const long long x = (long long)((unsigned long long)(uint32_t)s << 16) + q;
    const uint32_t top = (uint32_t)(s >> 32) + (uint32_t)(x >> 48);
    const double B = __hiloint2double(0x46300000, (int)(top ^ 0x80000000u));
    const double A = __hiloint2double(0x43300000 | (int)((x >> 32) & 0xffff), (int)x);
    return (B - 0x1.000008000001p+100) + A;  // 2^100 + 2^79 + 2^52
}
// r 2^(E - 2114) where r is 0 or the result leaves the normal numbers
__device__ __noinline__ double scale80_far(double r, int E) {
    const int hi = __double2hiint(r), e = (hi >> 20) & 0x7ff;
    if (e == 0) return 0.0;
    const double f = scale_far(((unsigned long long)__double_as_longlong(r) & 0xfffffffffffffull) | (1ull << 52),
                               e + E - 2114);
    return hi < 0 ? -f : f;
}
// Eight of them.  Branch-free but for one rare test of all eight: a branch per element kept
// the elements' latencies from overlapping (750 cycles each).
__device__ __forceinline__ void round80(const long long* s, const float (&v0)[8], const float (&v1)[8],
                                        const int (&E)[8], double (&r)[8]) {
    uint32_t far = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        r[j] = significand80(s[j], (long long)__float2int_rn(v0[j]) * 256 + __float2int_rn(v1[j]));
    double n[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int hi = __double2hiint(r[j]), e = (hi >> 20) & 0x7ff;
        far |= (uint32_t)(e + E[j] - 2115) >= 2046u || e == 0 ? 1u << j : 0u;
        n[j] = __hiloint2double(hi + ((E[j] - 2114) << 20), __double2loint(r[j]));
    }
    if (far) {
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
            if (!(far >> j & 1)) continue;
            double x = r[0];
            int Ej = E[0];
#pragma unroll
            for (int u = 1; u < 8; ++u) {
                x = j == u ? r[u] : x;
                Ej = j == u ? E[u] : Ej;
            }
            const double f = scale80_far(x, Ej);
#pragma unroll
            for (int u = 0; u < 8; ++u) n[u] = j == u ? f : n[u];
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = n[j];
}

// SHORT: k16 <= HI_CHUNK
template <bool SHORT>
__global__ void __launch_bounds__(NTHREADS, 1) oz_gemm_kernel(const __grid_constant__ OzArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * STAGES), tempty0 = smem_u32(bars + 2 * STAGES + 2);
    const uint32_t done_bar = smem_u32(bars + 2 * STAGES + 4);
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 5);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = g.tiles_m * g.tiles_n * g.batch, k16 = g.k16, ng = n_groups(k16);
    int* const err = g.err;
    const long long wait = g.wait;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull0 + 8 * a, 1);
            mbar_init(tempty0 + 8 * a, 256);
        }
        mbar_init(done_bar, 1);
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
            const uint8_t* B = g.B + ((long long)tb * g.tiles_n + tn) * k16 * BLOCK;
            for (int q = 0; ok && q < ng; ++q) {
                const Group G = group_at(q, k16);
                const int sp = steps_per_stage(G.p);
                const uint32_t nb = (uint32_t)(2 * G.p + 2) * PLANE;
                for (int k = G.k0; k < G.k1; k += sp) {
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1, err, wait)) { ok = false; break; }
                    const int n = min(sp, G.k1 - k);
                    uint32_t dst = smem_u32(smem + s * STAGE);
                    const uint32_t fb = full0 + 8 * s;
                    mbar_expect_tx(fb, 2 * nb * n);
                    for (int u = 0; u < n; ++u) {
                        bulk_load(dst, A + (long long)(k + u) * BLOCK, nb, fb);
                        bulk_load(dst + nb, B + (long long)(k + u) * BLOCK, nb, fb);
                        dst += 2 * nb;
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
    } else if (warp == 1 && lane == 0) {
        // ---------------- MMA issuer
        int s = 0, acc = 0;
        uint32_t ph = 0, aph = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            for (int q = 0; ok && q < ng; ++q) {
                const Group G = group_at(q, k16);
                const int sp = steps_per_stage(G.p);
                const uint32_t nb = (uint32_t)(2 * G.p + 2) * PLANE;
                if (!mbar_wait(tempty0 + 8 * acc, aph ^ 1, err, wait)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(acc * 2 * TILE);
                for (int k = G.k0; k < G.k1; k += sp) {
                    if (!mbar_wait(full0 + 8 * s, ph, err, wait)) { ok = false; break; }
                    tc_fence_after();
                    const int n = min(sp, G.k1 - k);
                    uint32_t a0 = smem_u32(smem + s * STAGE);
                    for (int u = 0; u < n; ++u, a0 += 2 * nb) {
                        const bool first = k + u == G.k0;
                        if (G.p == 0) issue_step<0>(a0, d, first);
                        else if (G.p == 1) issue_step<1>(a0, d, first);
                        else if (G.p == 2) issue_step<2>(a0, d, first);
                        else issue_step<3>(a0, d, first);
                    }
                    mma_commit(empty0 + 8 * s);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                mma_commit(tfull0 + 8 * acc);
                if (++acc == 2) { acc = 0; aph ^= 1; }
            }
        }
        // all MMAs issued by this CTA complete before TMEM is released
        mma_commit(done_bar);
        const long long t0 = clock64();
        while (!mbar_try(done_bar, 0) && clock64() - t0 < DRAIN_CYCLES) {
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: row = TMEM lane, 64 columns per thread
        const int quarter = warp & 3, row = quarter * 32 + lane, col0 = ((warp - 2) >> 2) * 64;
        long long* const stash = SHORT ? nullptr : g.stash + (long long)blockIdx.x * (TILE * TILE) + col0 * TILE + row;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        int acc = 0;
        uint32_t aph = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            int tb, tm, tn;
            tile_at(g, t, tb, tm, tn);
            const int* const exA = g.exA + (long long)tb * g.tiles_m * TILE;
            const int* const exB = g.exB + (long long)tb * g.tiles_n * TILE;
            const int m = tm * TILE + row, n0 = tn * TILE + col0, nc = min(64, g.N - n0);
            const bool mine = m < g.M;
            // exponents: this thread's row, and two of the warp's 64 columns per lane
            const int Ea = mine ? exA[m] : 0;
            const int Eb0 = lane < nc ? exB[n0 + lane] : 0, Eb1 = lane + 32 < nc ? exB[n0 + 32 + lane] : 0;
            const bool special = __any_sync(0xffffffffu, Ea == 0x7ff || Eb0 == 0x7ff || Eb1 == 0x7ff);
            const int ea = max(Ea, 1);
            double* const Cm = g.C + tb * g.cb + m + (long long)n0 * g.ldc;
            const double alpha = g.alpha, beta = g.beta;
            long long sum[64];
#pragma unroll
            for (int j = 0; j < 64; ++j) sum[j] = 0;
            // The read-out walks the columns eight at a time in a rolled loop, the sums moving
            // down by eight registers each turn: unrolled it outgrew the instruction cache and
            // took 70 us a tile.
            // C += v goes to L2 as a reduction (one per element, IEEE rounding): reading C
            // here left the warps waiting on its loads for two thirds of the read-out.
            const int flip = alpha == -1.0 ? 0x80000000 : 0;
            const bool plain = (alpha == 1.0 || alpha == -1.0) && (beta == 0.0 || beta == 1.0), add = beta == 1.0;
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
                        double* const p = Cm + (long long)(c + j) * g.ldc;
                        double v = r[0];
#pragma unroll
                        for (int u = 1; u < 8; ++u) v = j == u ? r[u] : v;
                        *p = beta == 0.0 ? alpha * v : fma(alpha, v, beta * *p);
                    }
                }
            };
            auto exps = [&](int c) { return ea + max(__shfl_sync(0xffffffffu, c < 32 ? Eb0 : Eb1, c & 31), 1); };
            auto rotate = [&]() {
#pragma unroll
                for (int j = 0; j < 56; ++j) sum[j] = sum[j + 8];
            };
            for (int q = 0; q < ng; ++q) {
                const Group G = group_at(q, k16);
                const bool straight = SHORT && G.last && !special;
                // the whole warp stays or leaves: tcgen05.ld is warp-collective
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, aph, err, wait));
                if (!ok) break;
                tc_fence_after();
                const uint32_t base = tmem_base + lanes + (uint32_t)(acc * 2 * TILE + col0);
                if (SHORT && G.last) {
#pragma unroll 1
                    for (int c = 0; straight && c < 64; c += 8) {
                        float v0[8], v1[8];
                        tmem_ld8x2(base + c, base + TILE + c, v0, v1);
                        double r[8];
                        int E[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) E[j] = exps(c + j);
                        round80(sum, v0, v1, E, r);
                        finish(c, r);
                        rotate();
                    }
                } else {
                    // weights of the two accumulators within the sums
                    const int w1 = (G.p & 1) || (SHORT && G.p == 2) ? 1 : 1 << 16, w0 = w1 << 8;
                    if (SHORT && G.p == 2)
#pragma unroll
                        for (int j = 0; j < 64; ++j) sum[j] <<= 16;
#pragma unroll
                    for (int c = 0; c < 64; c += 16) {
                        float v[16];
                        tmem_ld16(base + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[c + j] += (long long)__float2int_rn(v[j]) * w0;
                        tmem_ld16(base + TILE + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[c + j] += (long long)__float2int_rn(v[j]) * w1;
                    }
                }
                tc_fence_before();
                mbar_arrive(tempty0 + 8 * acc);
                if (++acc == 2) { acc = 0; aph ^= 1; }
                if (!SHORT && G.last_hi) {
#pragma unroll
                    for (int j = 0; j < 64; ++j) {
                        stash[j * TILE] = sum[j];
                        sum[j] = 0;
                    }
                }
            }
            if (!ok) break;
            if (!SHORT && !special) {
#pragma unroll 1
                for (int c = 0; c < 64; c += 8) {
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
                // an infinity or a NaN in these rows or columns: plain sums, or NaN where C
                // takes the place of B
                for (int c = 0; c < nc; ++c) {
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
        CUDA_CHECK(cudaFuncSetAttribute(oz_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        CUDA_CHECK(cudaFuncSetAttribute(oz_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        CUDA_CHECK(cudaFuncSetAttribute(oz_split_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM));
    });
}

void OzMat::split(const double* a, long long rs_, long long ks_, int rows_, int k_, cudaStream_t st, int batch_,
                  long long bs_) {
    set_up();
    rows = rows_;
    k = k_;
    k16 = ceil_div(k, 16);
    batch = batch_;
    src = a;
    rs = rs_;
    ks = ks_;
    bs = bs_;
    const int rb = ceil_div(rows, TILE), eb = rb * TILE;
    d.alloc((size_t)batch * rb * k16 * (BLOCK / 16), st);
    ex.alloc((size_t)batch * eb, st);
    if (k <= FUSED_K && (rs == 1 || ks == 1)) {
        LAUNCH(oz_split_fused, dim3(ceil_div(rows, 32), 1, batch), 256, k16 * 16 * 33 * 8, st, a, rs, ks, rows, k, k16,
               ex.get(), d.get(), bs, eb);
        return;
    }
    if (ks == 1) {
        LAUNCH(oz_exponent_cols, dim3(ceil_div(rows, 8), 1, batch), 256, 0, st, a, rs, rows, k, ex.get(), bs, eb);
    } else {
        ex.zero();
        const int kper = 32;
        LAUNCH(oz_exponent_rows, dim3(rb, ceil_div(k, kper), batch), TILE, 0, st, a, rs, ks, rows, k, kper, ex.get(), bs,
               eb);
    }
    // about four CTAs per SM's worth of k16 steps
    const int gy = std::max(1, std::min(k16, 152 * 8 / (rb * batch)));
    LAUNCH(oz_split, dim3(rb, gy, batch), dim3(TILE, 2), 0, st, a, rs, ks, rows, k, k16, ex.get(), d.get(), bs, eb);
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
    g.tiles_n = ceil_div(g.N, TILE);
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
    const bool brief = g.k16 <= HI_CHUNK;
    DevBuf<long long> stash(brief ? 0 : (size_t)grid * TILE * TILE, st);
    g.stash = stash.get();
    g.err = err;
    g.wait = gemm_wait_cycles();
    // credited as BF16 tensor work: 36 digit products
    const double fl = 72.0 * g.batch * g.M * g.N * g.K,
                 by = g.batch * (16.0 * ((double)g.M + g.N) * g.K + (beta == 0.0 ? 8.0 : 16.0) * g.M * g.N);
    if (brief) TIMED_LAUNCH("oz_gemm", fl, by, oz_gemm_kernel<true>, grid, NTHREADS, SMEM_BYTES, st, g);
    else TIMED_LAUNCH("oz_gemm", fl, by, oz_gemm_kernel<false>, grid, NTHREADS, SMEM_BYTES, st, g);
}

}  // namespace sqbem
