// tube_fourier.cu -- Fourier blocks of the tube and solves through them (see
// tube_fourier.cuh).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <vector>

#include "common.cuh"
#include "packed.cuh"
#include "tc_gemm.cuh"
#include "tube_fourier.cuh"

namespace cg = cooperative_groups;

namespace sqbem {

namespace {

constexpr int FT_MAXF = FT_MAX_SECTORS / 2 + 1;  // frequencies held at most
constexpr int FT_JOBS = 48;                      // jobs per grouped launch
constexpr double TWO_PI = 6.283185307179586476925286766559;

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ---------------------------------------------------------------- the blocks
// C^_f[(a, al), (b, be)] = sum_d w^{f d} sum_g T0[3 a + al, 3 panel(b, d) + g] R_d[g][be],
// accumulated in FP64 (high frequencies cancel), stored as FP32 complex.
// Thread: row r = (a, al); blockIdx.y: column c = (b, be); blockIdx.z: job.
struct ChatJob {
    const float* T0;
    const int* panel;
    float2* C;  // nf blocks of n3 x n3, column-major
};
struct ChatArgs {
    int n;
    int nth, nb, nf;
    double2 tw[FT_MAX_SECTORS];  // (cos, sin) of 2 pi k / nth
    ChatJob j[FT_JOBS];
};

__global__ void chat_kernel(const __grid_constant__ ChatArgs args) {
    const ChatJob& J = args.j[blockIdx.z];
    const int nth = args.nth, n3 = 3 * args.nb;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n3) return;
    const int c = blockIdx.y, b = c / 3, be = c % 3;
    double re[FT_MAXF], im[FT_MAXF];
#pragma unroll
    for (int f = 0; f < FT_MAXF; ++f) re[f] = im[f] = 0.0;
    for (int d = 0; d < nth; ++d) {
        const int q = J.panel[b * nth + d];
        const float* col = J.T0 + r + (long long)(3 * q) * n3;
        const double cs = args.tw[d].x, sn = args.tw[d].y;
        double v;  // (T0 R_d)[r, 3 q + be]
        if (be == 2) v = col[2LL * n3];
        else if (be == 0) v = cs * col[0] + sn * col[n3];
        else v = -sn * col[0] + cs * col[n3];
        int k = 0;  // f d mod nth
#pragma unroll
        for (int f = 0; f < FT_MAXF; ++f) {
            if (f < args.nf) {
                re[f] += v * args.tw[k].x;
                im[f] += v * args.tw[k].y;
                k += d;
                if (k >= nth) k -= nth;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < FT_MAXF; ++f)
        if (f < args.nf) J.C[(long long)f * n3 * n3 + (long long)c * n3 + r] = make_float2((float)re[f], (float)im[f]);
}

// ---------------------------------------------------------------- inversion
// In-place Gauss-Jordan inversion with partial pivoting of one n x n complex block per
// cluster of CL CTAs.  The block lives in registers: CTA q holds the columns
// [q w, q w + w), warp v of it the columns q w + v + 16 j (j < CJ), lane l the rows
// l + 32 i (i < RI).  Rows are not exchanged: the pivot row of step k is the row p_k with the
// largest |a_ik| among those that have not been one, and the permutation is applied when the
// inverse is written, A^-1[k, p_j] = a[p_k, j].
//   Step k: column k and p_k come from the shared memory of the CTA, where the warp that holds
// the column has put them in every CTA of the cluster; each warp passes its part of row p_k
// around through shared memory and eliminates column k from its own columns.  The warp that
// holds column k + 1 eliminates that one first, finds p_{k+1} and sends both off before it goes
// on, so that the exchange runs during the elimination.  A zero pivot sets bit 1 of *flag.
//   With the block in shared memory every step read and wrote all of it there (1900 clocks at
// 128 bytes per clock for n = 174 in two CTAs, against 500 of FP32 arithmetic).  Now the
// exchange bounds a step (about 1 us): 277 blocks of order 162 .. 174 in two CTAs each
// 1575 -> 739 us, one tube's 13 blocks in eight 324 -> 158 us.
constexpr int GJ_WARPS = 16, GJ_THREADS = 32 * GJ_WARPS;
constexpr int GJ_MAXB = 1024;
struct GjArgs {
    int n, w, nblk;
    int* flag;
    float2* C[GJ_MAXB];
};

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// (re, im) -= (mr, mi) r for two rows; a negated half rounds like the product it replaces
__device__ __forceinline__ void eliminate(uint64_t& re, uint64_t& im, uint64_t mr, uint64_t mi, float2 r) {
    const uint64_t rx = pack2(r.x, r.x), ry = pack2(r.y, r.y), nry = pack2(-r.y, -r.y);
    re = sub2(re, fma2(mr, rx, mul2(mi, nry)));
    im = sub2(im, fma2(mr, ry, mul2(mi, rx)));
}

template <int RI, int CJ, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(GJ_THREADS, 1) gj_kernel(const __grid_constant__ GjArgs args) {
    cg::cluster_group cl = cg::this_cluster();
    constexpr int RP = RI / 2, NR = 32 * RI;
    __shared__ float2 colk[2][NR];           // column k, double-buffered
    __shared__ int meta[2];                  // p_k (-1: zero pivot)
    __shared__ float2 rowk[GJ_WARPS][CJ];    // a warp's part of row p_k
    __shared__ int piv[NR], pos[NR];         // p_k, and its inverse
    const int n = args.n, w = args.w, rank = (int)cl.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = rank * w, wl = max(0, min(w, n - c0));
    float2* const C = args.C[blockIdx.x / CL];
    // packed by pairs of rows: lane + 64 i and lane + 64 i + 32
    uint64_t re[RP][CJ], im[RP][CJ];
    unsigned done = 0;  // bit i: row lane + 32 i has been a pivot row (or is past the block)
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int r = lane + 64 * i;
        if (r >= n) done |= 1u << 2 * i;
        if (r + 32 >= n) done |= 2u << 2 * i;
#pragma unroll
        for (int j = 0; j < CJ; ++j) {
            const int c = warp + GJ_WARPS * j;
            const float2* const src = C + (long long)(c0 + c) * n + r;
            const float2 x = r < n && c < wl ? src[0] : make_float2(0.f, 0.f);
            const float2 y = r + 32 < n && c < wl ? src[32] : make_float2(0.f, 0.f);
            re[i][j] = pack2(x.x, y.x);
            im[i][j] = pack2(x.y, y.y);
        }
    }
    // column k (this lane's rows) and its pivot row into every CTA; by the whole warp that holds it
    const auto publish = [&](int k, const uint64_t (&vr)[RP], const uint64_t (&vi)[RP]) {
        float2 v[2 * RP];
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const float2 x = unpack2(vr[i]), y = unpack2(vi[i]);
            v[2 * i] = make_float2(x.x, y.x);
            v[2 * i + 1] = make_float2(x.y, y.y);
        }
        unsigned best = 0;
        unsigned mag[2 * RP];
#pragma unroll
        for (int i = 0; i < 2 * RP; ++i) {
            const float m = v[i].x * v[i].x + v[i].y * v[i].y;
            mag[i] = (done >> i & 1) || !(m > 0.f) ? 0u : __float_as_uint(m);
            best = max(best, mag[i]);
        }
        best = __reduce_max_sync(0xffffffffu, best);
        unsigned row = 0x7fffffffu;
#pragma unroll
        for (int i = 2 * RP - 1; i >= 0; --i)
            if (mag[i] == best) row = lane + 32 * i;
        row = __reduce_min_sync(0xffffffffu, row);
#pragma unroll
        for (int q = 0; q < CL; ++q) {
            float2* const dst = cl.map_shared_rank(&colk[k & 1][0], q);
#pragma unroll
            for (int i = 0; i < 2 * RP; ++i) dst[lane + 32 * i] = v[i];
        }
        if (lane < CL) *cl.map_shared_rank(&meta[k & 1], lane) = best ? (int)row : -1;
    };
    cl.sync();  // every CTA of the cluster runs before its shared memory is written
    if (rank == 0 && warp == 0) {
        uint64_t vr[RP], vi[RP];
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            vr[i] = re[i][0];
            vi[i] = im[i][0];
        }
        publish(0, vr, vi);
    }
    cluster_arrive();
    bool bad = false;
    for (int k = 0; k < n; ++k) {
        cluster_wait();
        const int p = meta[k & 1];
        if (p < 0) { bad = true; break; }  // the same in every CTA of the cluster
        const int lp = p & 31, ip = p >> 5;
        const float2 pv = colk[k & 1][p];
        uint64_t mr[RP], mi[RP];
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const float2 x = colk[k & 1][lane + 64 * i], y = colk[k & 1][lane + 64 * i + 32];
            mr[i] = pack2(x.x, y.x);
            mi[i] = pack2(x.y, y.y);
        }
        if (threadIdx.x == 0) piv[k] = p;
        const float s2 = 1.f / (pv.x * pv.x + pv.y * pv.y);
        const float2 d = make_float2(pv.x * s2, -pv.y * s2);  // 1 / pivot
        // column k of the inverse: -m_i / pivot, and 1 / pivot in row p: the elimination of zeros
        const int own = k - c0, j0 = own >= 0 && own < wl && (own & (GJ_WARPS - 1)) == warp ? own / GJ_WARPS : -1;
        if (j0 >= 0) {
#pragma unroll
            for (int j = 0; j < CJ; ++j)
                if (j == j0) {
#pragma unroll
                    for (int i = 0; i < RP; ++i) re[i][j] = im[i][j] = 0;
                }
        }
        if (lane == lp) {
#pragma unroll
            for (int h = 0; h < 2 * RP; ++h)
                if (h == ip) {
                    const int i = h >> 1, odd = h & 1;
#pragma unroll
                    for (int j = 0; j < CJ; ++j) {
                        const float2 x = unpack2(re[i][j]), y = unpack2(im[i][j]);
                        float2 r = cmul(odd ? make_float2(x.y, y.y) : make_float2(x.x, y.x), d);
                        if (j == j0) r = d;
                        re[i][j] = odd ? pack2(x.x, r.x) : pack2(r.x, x.y);
                        im[i][j] = odd ? pack2(y.x, r.y) : pack2(r.y, y.y);
                        rowk[warp][j] = r;
                    }
                    const float2 x = unpack2(mr[i]), y = unpack2(mi[i]);
                    mr[i] = odd ? pack2(x.x, 0.f) : pack2(0.f, x.y);
                    mi[i] = odd ? pack2(y.x, 0.f) : pack2(0.f, y.y);
                }
            done |= 1u << ip;
        }
        __syncwarp();
        if (k + 1 < n) {
            const int nx = k + 1 - c0;
            if (nx >= 0 && nx < wl && (nx & (GJ_WARPS - 1)) == warp) {
                const int j1 = nx / GJ_WARPS;
                const float2 rk = rowk[warp][j1];
                uint64_t vr[RP], vi[RP];
#pragma unroll
                for (int j = 0; j < CJ; ++j)
                    if (j == j1) {
#pragma unroll
                        for (int i = 0; i < RP; ++i) {
                            vr[i] = re[i][j];
                            vi[i] = im[i][j];
                        }
                    }
#pragma unroll
                for (int i = 0; i < RP; ++i) eliminate(vr[i], vi[i], mr[i], mi[i], rk);
                publish(k + 1, vr, vi);
            }
            // this step's column has been read, the next one's sent: buffer k & 1 is free for k + 2
            cluster_arrive();
        }
#pragma unroll
        for (int j = 0; j < CJ; ++j) {
            const float2 rk = rowk[warp][j];
#pragma unroll
            for (int i = 0; i < RP; ++i) eliminate(re[i][j], im[i][j], mr[i], mi[i], rk);
        }
        __syncwarp();  // rowk is written again in the next step
    }
    if (bad) {
        if (threadIdx.x == 0 && rank == 0) atomicOr(args.flag, 2);
        return;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += GJ_THREADS) pos[piv[k]] = k;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
        const int c = warp + GJ_WARPS * j;
        if (c >= wl) continue;
        float2* const dst = C + (long long)piv[c0 + c] * n;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const float2 x = unpack2(re[i][j]), y = unpack2(im[i][j]);
            const int r = lane + 64 * i;
            if (r < n) dst[pos[r]] = make_float2(x.x, y.x);
            if (r + 32 < n) dst[pos[r + 32]] = make_float2(x.y, y.y);
        }
    }
}

// Columns per CTA and CTAs per block for n <= 256: a thread's part of the block has to stay
// in its registers (at most 36 complex entries).  One tube's blocks (13 for 24 sectors) go to
// clusters of eight, which still leave SMs free.
struct GjShape {
    int ri, cl;
};
GjShape gj_shape(int n, int nblk) {
    const int ri = n <= 128 ? 4 : n <= 192 ? 6 : 8;
    return {ri, nblk * 8 <= 152 ? 8 : ri == 8 ? 4 : 2};
}

void launch_gj(GjArgs& g, cudaStream_t st) {
    if (g.n > 256) fail(SQBEM_ERR_ARG, "Gauss-Jordan: block order %d too large", g.n);
    const GjShape s = gj_shape(g.n, g.nblk);
    g.w = (g.n + s.cl - 1) / s.cl;
    // credited: 8 n^3 FP32 flops per complex inversion; bytes: the block read and written
    const double fl = 8.0 * g.nblk * (double)g.n * g.n * g.n, by = 16.0 * g.nblk * (double)g.n * g.n;
    const int grid = s.cl * g.nblk;
#define GJ_LAUNCH(RI, CJ, CL) TIMED_LAUNCH("fourier_inverse", fl, by, (gj_kernel<RI, CJ, CL>), grid, GJ_THREADS, 0, st, g)
    if (s.ri == 4 && s.cl == 8) GJ_LAUNCH(4, 1, 8);
    else if (s.ri == 4) GJ_LAUNCH(4, 4, 2);
    else if (s.ri == 6 && s.cl == 8) GJ_LAUNCH(6, 2, 8);
    else if (s.ri == 6) GJ_LAUNCH(6, 6, 2);
    else if (s.cl == 8) GJ_LAUNCH(8, 2, 8);
    else GJ_LAUNCH(8, 4, 4);
#undef GJ_LAUNCH
}

// The real form [[Re, -Im], [Im, Re]] of every inverse (n x n complex,
// column-major) as split BF16, row-major with leading dimension ldk, through
// 32 x 32 shared-memory tiles: reads along the source columns, writes along the
// destination rows.  blockIdx.z: block.
struct RfArgs {
    int n, ldk, nblk;
    const float2* C[GJ_MAXB];
    bf16* hi[GJ_MAXB];
    bf16* lo[GJ_MAXB];
};

__global__ void realform_kernel(const __grid_constant__ RfArgs args) {
    __shared__ float tile[32][33];
    const int n = args.n, m2 = 2 * n;
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;  // tile of the real form
    const float2* C = args.C[blockIdx.z];
    // load: element (r, c) of the real form, r = r0 + tx, c = c0 + ty + 8 q
    for (int q = 0; q < 4; ++q) {
        const int r = r0 + threadIdx.x, c = c0 + threadIdx.y + 8 * q;
        float v = 0.f;
        if (r < m2 && c < m2) {
            const int rr = r < n ? r : r - n, cc = c < n ? c : c - n;
            const float2 x = C[(long long)cc * n + rr];
            v = (r < n) == (c < n) ? x.x : (r < n ? -x.y : x.y);
        }
        tile[threadIdx.y + 8 * q][threadIdx.x] = v;
    }
    __syncthreads();
    // store: row r = r0 + ty + 8 q, column c = c0 + tx
    bf16* H = args.hi[blockIdx.z];
    bf16* L = args.lo[blockIdx.z];
    for (int q = 0; q < 4; ++q) {
        const int r = r0 + threadIdx.y + 8 * q, c = c0 + threadIdx.x;
        if (r < m2 && c < m2) {
            const float v = tile[threadIdx.x][threadIdx.y + 8 * q];
            const bf16 h = __float2bfloat16_rn(v);
            H[(long long)r * args.ldk + c] = h;
            L[(long long)r * args.ldk + c] = __float2bfloat16_rn(v - __bfloat162float(h));
        }
    }
}

// ---------------------------------------------------------------- transforms
// Forward: X^_f[(a, al), j] = (1 / nth) sum_s w^{-f s} (R_s^T x_{panel(a, s)})_al for
// column j, written as the split column-major operand of the frequency's GEMM:
// rows [0, n3) the real parts, [n3, 2 n3) the imaginary parts, leading dimension
// ldk, one plane of ldk x nc per frequency.  Thread: r = (a, al); blockIdx.x:
// column; blockIdx.y: job.
struct DftJob {
    const int* panel;
    const float2* tw;
    const void* x;  // forward: input X; inverse: the GEMM result Y^
    long long ldx;
    void* y;        // forward: unused; inverse: output Y
    long long ldy;
    bf16* h;        // forward: X^ split; inverse: optional split copy of Y, element
    bf16* l;        // (r, j) at r * hrs + j * hcs
    long long hrs, hcs;
    int nc, nb, nth, nf, ldk;
};
struct DftArgs {
    int n;
    float2 tw[FT_MAX_SECTORS];  // (cos, sin) of 2 pi k / nth (the kernels specialised on nth read these)
    DftJob j[FT_JOBS];
};

template <class TI>
__global__ void __launch_bounds__(192) fdft_kernel(const __grid_constant__ DftArgs args) {
    const DftJob& J = args.j[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= J.nc) return;
    const int n3 = 3 * J.nb, nth = J.nth, nf = J.nf;
    const TI* x = reinterpret_cast<const TI*>(J.x) + (long long)j * J.ldx;
    const float scale = 1.f / (float)nth;
    for (int r = threadIdx.x; r < n3; r += blockDim.x) {
        const int a = r / 3, al = r - 3 * a;
        float re[FT_MAXF], im[FT_MAXF];
#pragma unroll
        for (int f = 0; f < FT_MAXF; ++f) re[f] = im[f] = 0.f;
        for (int s = 0; s < nth; ++s) {
            const int p = J.panel[a * nth + s];
            const float2 rs = J.tw[s];
            float v;  // (R_s^T x_p)_al
            if (al == 2) v = (float)x[3 * p + 2];
            else {
                const float x0 = (float)x[3 * p], x1 = (float)x[3 * p + 1];
                v = al == 0 ? rs.x * x0 + rs.y * x1 : -rs.y * x0 + rs.x * x1;
            }
            int k = 0;  // f s mod nth
#pragma unroll
            for (int f = 0; f < FT_MAXF; ++f) {
                if (f < nf) {
                    const float2 t = J.tw[k];
                    re[f] += v * t.x;
                    im[f] -= v * t.y;
                    k += s;
                    if (k >= nth) k -= nth;
                }
            }
        }
#pragma unroll
        for (int f = 0; f < FT_MAXF; ++f) {
            if (f < nf) {
                const long long o = ((long long)f * J.nc + j) * J.ldk;
                const float vr = re[f] * scale, vi = im[f] * scale;
                const bf16 hr = __float2bfloat16_rn(vr), hi = __float2bfloat16_rn(vi);
                J.h[o + r] = hr;
                J.l[o + r] = __float2bfloat16_rn(vr - __bfloat162float(hr));
                J.h[o + n3 + r] = hi;
                J.l[o + n3 + r] = __float2bfloat16_rn(vi - __bfloat162float(hi));
            }
        }
    }
}

// Inverse: y~_s = sum over all frequencies of w^{f s} y^_f = Re y^_0 + 2 sum_{0 < f < nth/2}
// Re(w^{f s} y^_f) (+ Re((-1)^s y^_{nth/2}) for even nth), then y_panel(a, s) = R_s y~_s.
// Y^ is the FP32 GEMM result: per frequency ldk x nc, column-major, rows [0, n3)
// real, [n3, 2 n3) imaginary.  Thread: representative a (strided); blockIdx.x:
// column; blockIdx.y: job.
template <class TO>
__global__ void __launch_bounds__(64) idft_kernel(const __grid_constant__ DftArgs args) {
    const DftJob& J = args.j[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= J.nc) return;
    const int n3 = 3 * J.nb, nth = J.nth, nf = J.nf;
    const float* yh = reinterpret_cast<const float*>(J.x) + (long long)j * J.ldk;
    const long long plane = (long long)J.nc * J.ldk;
    TO* y = reinterpret_cast<TO*>(J.y) + (long long)j * J.ldy;
    const bool even = (nth & 1) == 0;
    // components 0 and 1 (rotated together), then component 2
    for (int a = threadIdx.x; a < J.nb; a += blockDim.x)
    for (int pass = 0; pass < 2; ++pass) {
        float r0[FT_MAXF], i0[FT_MAXF], r1[FT_MAXF], i1[FT_MAXF];
#pragma unroll
        for (int f = 0; f < FT_MAXF; ++f) {
            r0[f] = i0[f] = r1[f] = i1[f] = 0.f;
            if (f < nf) {
                const float wgt = (f == 0 || (even && 2 * f == nth)) ? 1.f : 2.f;
                const float* pf = yh + f * plane;
                if (pass == 0) {
                    r0[f] = wgt * pf[3 * a];
                    i0[f] = wgt * pf[n3 + 3 * a];
                    r1[f] = wgt * pf[3 * a + 1];
                    i1[f] = wgt * pf[n3 + 3 * a + 1];
                } else {
                    r0[f] = wgt * pf[3 * a + 2];
                    i0[f] = wgt * pf[n3 + 3 * a + 2];
                }
            }
        }
        for (int s = 0; s < nth; ++s) {
            float v0 = 0.f, v1 = 0.f;
            int k = 0;
#pragma unroll
            for (int f = 0; f < FT_MAXF; ++f) {
                if (f < nf) {
                    const float2 t = J.tw[k];
                    v0 += t.x * r0[f] - t.y * i0[f];
                    if (pass == 0) v1 += t.x * r1[f] - t.y * i1[f];
                    k += s;
                    if (k >= nth) k -= nth;
                }
            }
            const int p = J.panel[a * nth + s];
            const float2 rs = J.tw[s];
            float o[2];
            int nout;
            long long row;
            if (pass == 0) {
                o[0] = rs.x * v0 - rs.y * v1;
                o[1] = rs.y * v0 + rs.x * v1;
                nout = 2;
                row = 3LL * p;
            } else {
                o[0] = v0;
                nout = 1;
                row = 3LL * p + 2;
            }
            for (int q = 0; q < nout; ++q) {
                y[row + q] = (TO)o[q];
                if (J.h) {
                    const long long e = (row + q) * J.hrs + (long long)j * J.hcs;
                    const bf16 h = __float2bfloat16_rn(o[q]);
                    J.h[e] = h;
                    J.l[e] = __float2bfloat16_rn(o[q] - __bfloat162float(h));
                }
            }
        }
    }
}

// Both transforms with the number of sectors known at compile time: the sector and frequency
// loops unrolled, the twiddles constant operands of the multiply-adds.  A CTA holds one column
// (blockIdx.x; job: blockIdx.y), whose rows by panel go through shared memory: they are
// 12-byte pieces there, gathered at the panels' numbers, and whole lines in global memory.
constexpr int FDFT_THREADS = 256, IDFT_THREADS = 96;
static_assert(FDFT_THREADS >= FT_MAX_ORDER && 3 * IDFT_THREADS >= FT_MAX_ORDER, "a CTA holds one column");
int fdft_threads(int nb) { return (3 * nb + 31) / 32 * 32; }
int idft_threads(int nb) { return nb <= 64 ? 64 : IDFT_THREADS; }
size_t dft_smem(int nth, int nb) { return (size_t)3 * nb * nth * sizeof(float); }

// Forward: a thread per row (a, c) of the spectrum, so that the 2-byte stores of a warp are
// contiguous.  A thread per representative with all three components held 164 registers for
// twelve warps per SM, which waited on its gathers: 265 us for 24 sectors, 54 representatives
// and 23040 columns, 206 here (111 at the copy's rate).
template <int NTH, class TI>
__global__ void __launch_bounds__(FDFT_THREADS) fdft_rep(const __grid_constant__ DftArgs args) {
    constexpr int NF = NTH / 2 + 1;
    const DftJob& J = args.j[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= J.nc) return;
    extern __shared__ __align__(16) float xs[];
    const int n3 = 3 * J.nb, nt = n3 * NTH, r = threadIdx.x, bd = blockDim.x;
    const TI* x = reinterpret_cast<const TI*>(J.x) + (long long)j * J.ldx;
    const float scale = 1.f / (float)NTH;
    // eight loads in flight per thread (a rolled remainder waited for each)
    int e0 = 0;
    if (sizeof(TI) == 4 && ((uintptr_t)x & 15) == 0) {
        for (int e = threadIdx.x; e < nt / 4; e += 8 * bd) {
            float4 q[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (e + u * bd < nt / 4) q[u] = __ldg(reinterpret_cast<const float4*>(x) + e + u * bd);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (e + u * bd < nt / 4) reinterpret_cast<float4*>(xs)[e + u * bd] = q[u];
        }
        e0 = nt & ~3;
    }
    for (int e = e0 + threadIdx.x; e < nt; e += 8 * bd) {
        TI q[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (e + u * bd < nt) q[u] = __ldg(x + e + u * bd);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (e + u * bd < nt) xs[e + u * bd] = (float)q[u];
    }
    __syncthreads();
    if (r >= n3) return;
    const int a = r / 3, c = r - 3 * a;
    const int* pa = J.panel + a * NTH;
    float v[NTH];  // component c of R_s^T x_{panel(a, s)}
#pragma unroll
    for (int s = 0; s < NTH; ++s) {
        const float* xp = xs + 3 * __ldg(pa + s);
        const float cs = args.tw[s].x, sn = args.tw[s].y;
        // c = 0: cs x0 + sn x1; c = 1: cs x1 - sn x0
        const float xa = xp[c], xb = xp[c == 0 ? 1 : 0];
        const float w = __fmaf_rn(cs, xa, __fmul_rn(c == 0 ? sn : -sn, xb));
        v[s] = c == 2 ? xa : w;
    }
    float re[NF], im[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        re[f] = v[0];
        im[f] = 0.f;
    }
    // sectors s and NTH - s: shared cosines, opposite sines
#pragma unroll
    for (int s = 1; 2 * s < NTH; ++s) {
        const float sum = v[s] + v[NTH - s], dif = v[s] - v[NTH - s];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            re[f] += sum * args.tw[(f * s) % NTH].x;
            im[f] -= dif * args.tw[(f * s) % NTH].y;
        }
    }
    if ((NTH & 1) == 0) {
#pragma unroll
        for (int f = 0; f < NF; ++f) re[f] += (f & 1) ? -v[NTH / 2] : v[NTH / 2];
    }
    const long long step = (long long)J.nc * J.ldk;
    bf16* h = J.h + (long long)j * J.ldk + r;
    bf16* l = J.l + (long long)j * J.ldk + r;
#pragma unroll
    for (int f = 0; f < NF; ++f, h += step, l += step) {
        const float vr = re[f] * scale, vi = im[f] * scale;
        const bf16 hr = __float2bfloat16_rn(vr), hi = __float2bfloat16_rn(vi);
        h[0] = hr;
        l[0] = __float2bfloat16_rn(vr - __bfloat162float(hr));
        h[n3] = hi;
        l[n3] = __float2bfloat16_rn(vi - __bfloat162float(hi));
    }
}

// Inverse: a thread per representative a, whose three components' 6 NF spectrum values it
// holds (the rotation R_s needs no exchange), and the sectors s and NTH - s from one pair of
// sums,
//   y~_s = A_s - B_s and y~_{NTH-s} = A_s + B_s with A_s = sum_f cos(2 pi f s / NTH) y^r_f and
//   B_s = sum_f sin(2 pi f s / NTH) y^i_f.
// With a thread per component and the sector loop rolled (twiddles by their index, partners by
// shuffles) a column took 16,700 warp instructions, whose issue bound it: 443 us for the
// columns above, 213 here (164 at the copy's rate).
template <int NTH, class TO>
__global__ void __launch_bounds__(IDFT_THREADS) idft_rep(const __grid_constant__ DftArgs args) {
    constexpr int NF = NTH / 2 + 1;
    const DftJob& J = args.j[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= J.nc) return;
    extern __shared__ __align__(16) float ys[];
    const int nb = J.nb, n3 = 3 * nb, nt = n3 * NTH, a = threadIdx.x;
    const float* yh = reinterpret_cast<const float*>(J.x) + (long long)j * J.ldk;
    const long long plane = (long long)J.nc * J.ldk;
    if (a < nb) {
        float yr[3][NF], yi[3][NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const float wgt = (f == 0 || 2 * f == NTH) ? 1.f : 2.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                yr[c][f] = wgt * __ldg(yh + f * plane + 3 * a + c);
                yi[c][f] = wgt * __ldg(yh + f * plane + n3 + 3 * a + c);
            }
        }
        const int* pa = J.panel + a * NTH;
        auto emit = [&](int s, const float (&v)[3]) {
            const float cs = args.tw[s].x, sn = args.tw[s].y;
            float* const o = ys + 3 * __ldg(pa + s);
            o[0] = cs * v[0] - sn * v[1];
            o[1] = sn * v[0] + cs * v[1];
            o[2] = v[2];
        };
#pragma unroll
        for (int s = 0; 2 * s <= NTH; ++s) {
            float A[3] = {}, B[3] = {};
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    A[c] += args.tw[(f * s) % NTH].x * yr[c][f];
                    B[c] += args.tw[(f * s) % NTH].y * yi[c][f];
                }
            const float lo[3] = {A[0] - B[0], A[1] - B[1], A[2] - B[2]};
            emit(s, lo);
            if (s > 0 && 2 * s < NTH) {
                const float hi[3] = {A[0] + B[0], A[1] + B[1], A[2] + B[2]};
                emit(NTH - s, hi);
            }
        }
    }
    __syncthreads();
    TO* const y = reinterpret_cast<TO*>(J.y) + (long long)j * J.ldy;
    bf16* const h = J.h ? J.h + (long long)j * J.hcs : nullptr;
    bf16* const l = J.h ? J.l + (long long)j * J.hcs : nullptr;
    int e0 = 0;
    if (sizeof(TO) == 4 && ((uintptr_t)y & 15) == 0 && (!h || (J.hrs == 1 && (((uintptr_t)h | (uintptr_t)l) & 7) == 0))) {
        e0 = nt & ~3;
        for (int e = 4 * threadIdx.x; e < e0; e += 4 * blockDim.x) {
            const float4 o = *reinterpret_cast<const float4*>(ys + e);
            *reinterpret_cast<float4*>(y + e) = o;
            if (h) {
                const float q[4] = {o.x, o.y, o.z, o.w};
                uint2 hv, lv;
                bf16 *hp = reinterpret_cast<bf16*>(&hv), *lp = reinterpret_cast<bf16*>(&lv);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    hp[u] = __float2bfloat16_rn(q[u]);
                    lp[u] = __float2bfloat16_rn(q[u] - __bfloat162float(hp[u]));
                }
                *reinterpret_cast<uint2*>(h + e) = hv;
                *reinterpret_cast<uint2*>(l + e) = lv;
            }
        }
    }
    for (int e = e0 + threadIdx.x; e < nt; e += blockDim.x) {
        const float o = ys[e];
        y[e] = (TO)o;
        if (h) {
            const bf16 hv = __float2bfloat16_rn(o);
            h[e * J.hrs] = hv;
            l[e * J.hrs] = __float2bfloat16_rn(o - __bfloat162float(hv));
        }
    }
}

// C^_f in FP32 for a compile-time sector count (thread: row r; blockIdx.y: column)
template <int NTH>
__global__ void chat_nth(const __grid_constant__ ChatArgs args, const __grid_constant__ DftArgs tw) {
    constexpr int NF = NTH / 2 + 1;
    const ChatJob& J = args.j[blockIdx.z];
    const int n3 = 3 * args.nb;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n3) return;
    const int c = blockIdx.y, b = c / 3, be = c % 3;
    const int* pb = J.panel + b * NTH;
    float re[NF], im[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) re[f] = im[f] = 0.f;
#pragma unroll
    for (int d = 0; d < NTH; ++d) {
        const float* col = J.T0 + r + (long long)(3 * pb[d]) * n3;
        const float cs = tw.tw[d].x, sn = tw.tw[d].y;
        float v;  // (T0 R_d)[r, 3 q + be]
        if (be == 2) v = col[2LL * n3];
        else if (be == 0) v = cs * col[0] + sn * col[n3];
        else v = -sn * col[0] + cs * col[n3];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            re[f] += v * tw.tw[(f * d) % NTH].x;
            im[f] += v * tw.tw[(f * d) % NTH].y;
        }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) J.C[(long long)f * n3 * n3 + (long long)c * n3 + r] = make_float2(re[f], im[f]);
}

}  // namespace

bool fourier_supported(const TubeSymmetry& sym) {
    return sym.ok && sym.nth >= 2 && sym.nth <= FT_MAX_SECTORS && 3 * sym.nb <= FT_MAX_ORDER;
}

void gauss_jordan_blocks(float2* C, int nblk, int n3, int* flag, cudaStream_t st) {
    for (int b0 = 0; b0 < nblk; b0 += GJ_MAXB) {
        GjArgs g;
        g.n = n3;
        g.nblk = std::min(GJ_MAXB, nblk - b0);
        g.flag = flag;
        for (int b = 0; b < g.nblk; ++b) g.C[b] = C + (size_t)(b0 + b) * n3 * n3;
        launch_gj(g, st);
    }
}

void fourier_build(const std::vector<FourierTube*>& fts, const std::vector<const TubeSymmetry*>& syms,
                   const std::vector<const float*>& T0s, const MixedCtx& cx) {
    // tubes of equal sector count and block order go through the same launches
    std::map<std::pair<int, int>, std::vector<size_t>> by;
    for (size_t k = 0; k < fts.size(); ++k) {
        const TubeSymmetry& S = *syms[k];
        if (!fourier_supported(S)) fail(SQBEM_ERR_ARG, "fourier_build: tube outside the Fourier path's limits");
        FourierTube& F = *fts[k];
        F.nth = S.nth;
        F.nb = S.nb;
        F.nf = S.nth / 2 + 1;
        F.n3 = 3 * S.nb;
        F.m2 = 2 * F.n3;
        F.ldk = (F.m2 + 7) / 8 * 8;
        F.nt = 3 * S.nb * S.nth;
        F.panel.alloc(S.panel.size(), cx.st);
        F.panel.upload(S.panel.data(), S.panel.size());
        std::vector<float2> tw(S.nth);
        for (int i = 0; i < S.nth; ++i)
            tw[i] = make_float2((float)std::cos(TWO_PI * i / S.nth), (float)std::sin(TWO_PI * i / S.nth));
        F.tw.alloc(S.nth, cx.st);
        F.tw.upload(tw.data(), S.nth);
        const size_t rf = (size_t)F.nf * F.m2 * F.ldk;
        F.Ah.alloc(rf, cx.st);
        F.Al.alloc(rf, cx.st);
        by[{S.nth, S.nb}].push_back(k);
    }
    for (const auto& kv : by) {
        const int nth = kv.first.first, nb = kv.first.second, n3 = 3 * nb, nf = nth / 2 + 1;
        const std::vector<size_t>& ids = kv.second;
        DevBuf<float2> C(ids.size() * nf * (size_t)n3 * n3, cx.st);
        for (size_t i0 = 0; i0 < ids.size(); i0 += FT_JOBS) {
            ChatArgs a;
            a.n = (int)std::min<size_t>(FT_JOBS, ids.size() - i0);
            a.nth = nth; a.nb = nb; a.nf = nf;
            for (int d = 0; d < nth; ++d) a.tw[d] = make_double2(std::cos(TWO_PI * d / nth), std::sin(TWO_PI * d / nth));
            for (int q = 0; q < a.n; ++q) {
                const size_t k = ids[i0 + q];
                a.j[q] = {T0s[k], fts[k]->panel.get(), C.get() + (i0 + q) * nf * (size_t)n3 * n3};
            }
            const double cby = 4.0 * 9.0 * a.n * nb * (double)nb * nth + 8.0 * a.n * nf * (double)n3 * n3;
            const dim3 cg3(ceil_div(n3, 64), n3, a.n);
            DftArgs tw;
            for (int d = 0; d < nth; ++d)
                tw.tw[d] = make_float2((float)std::cos(TWO_PI * d / nth), (float)std::sin(TWO_PI * d / nth));
            if (nth == 24) TIMED_LAUNCH("fourier_inverse", 0.0, cby, chat_nth<24>, cg3, 64, 0, cx.st, a, tw);
            else if (nth == 30) TIMED_LAUNCH("fourier_inverse", 0.0, cby, chat_nth<30>, cg3, 64, 0, cx.st, a, tw);
            else if (nth == 36) TIMED_LAUNCH("fourier_inverse", 0.0, cby, chat_nth<36>, cg3, 64, 0, cx.st, a, tw);
            else TIMED_LAUNCH("fourier_inverse", 0.0, cby, chat_kernel, cg3, 64, 0, cx.st, a);
        }
        const int nblk_all = (int)(ids.size() * nf);
        for (int b0 = 0; b0 < nblk_all; b0 += GJ_MAXB) {
            GjArgs g;
            g.n = n3;
            g.nblk = std::min(GJ_MAXB, nblk_all - b0);
            g.flag = cx.flag;
            RfArgs r;
            r.n = n3;
            r.nblk = g.nblk;
            for (int b = 0; b < g.nblk; ++b) {
                const int gb = b0 + b;
                const size_t k = ids[gb / nf];
                const int f = gb % nf;
                g.C[b] = C.get() + (size_t)gb * n3 * n3;
                r.C[b] = g.C[b];
                r.hi[b] = fts[k]->Ah.get() + (size_t)f * fts[k]->m2 * fts[k]->ldk;
                r.lo[b] = fts[k]->Al.get() + (size_t)f * fts[k]->m2 * fts[k]->ldk;
                r.ldk = fts[k]->ldk;
            }
            launch_gj(g, cx.st);
            const int t = ceil_div(2 * n3, 32);
            TIMED_LAUNCH("fourier_inverse", 0.0, g.nblk * (8.0 * n3 * n3 + 16.0 * n3 * n3), realform_kernel,
                         dim3(t, t, g.nblk), dim3(32, 8), 0, cx.st, r);
        }
    }
}

void fourier_solve(const std::vector<FourierJob>& jobs, const MixedCtx& cx) {
    if (jobs.empty()) return;
    const bool in64 = jobs[0].x64 != nullptr, out64 = jobs[0].y64 != nullptr;
    for (const FourierJob& J : jobs)
        if ((J.x64 != nullptr) != in64 || (J.y64 != nullptr) != out64 || !J.ft)
            fail(SQBEM_ERR_ARG, "fourier_solve: mixed precisions in one call");
    // per job: X^ (split) and Y^ (FP32), nf planes of ldk x nc each
    std::vector<DevBuf<bf16>> xh(jobs.size()), xl(jobs.size());
    std::vector<DevBuf<float>> yh(jobs.size());
    for (size_t k = 0; k < jobs.size(); ++k) {
        const FourierTube& F = *jobs[k].ft;
        const size_t sz = (size_t)F.nf * F.ldk * jobs[k].nc;
        xh[k].alloc(sz, cx.st);
        xl[k].alloc(sz, cx.st);
        yh[k].alloc(sz, cx.st);
    }
    auto dft_job = [&](size_t k, bool forward) {
        const FourierJob& J = jobs[k];
        const FourierTube& F = *J.ft;
        DftJob d;
        d.panel = F.panel.get();
        d.tw = F.tw.get();
        d.nc = J.nc; d.nb = F.nb; d.nth = F.nth; d.nf = F.nf; d.ldk = F.ldk;
        if (forward) {
            d.x = in64 ? (const void*)J.x64 : (const void*)J.x32;
            d.ldx = J.ldx;
            d.y = nullptr; d.ldy = 0;
            d.h = xh[k].get(); d.l = xl[k].get(); d.hrs = 1; d.hcs = 0;
        } else {
            d.x = yh[k].get(); d.ldx = 0;
            d.y = out64 ? (void*)J.y64 : (void*)J.y32;
            d.ldy = J.ldy;
            d.h = J.yh; d.l = J.yl; d.hrs = J.srs; d.hcs = J.scs;
        }
        return d;
    };
    int maxnc = 0;
    for (const FourierJob& J : jobs) maxnc = std::max(maxnc, J.nc);
    // credited bytes of a transform: X (or Y) once, X^ (or Y^) once
    auto dft_bytes = [&](size_t i0, int n, bool forward) {
        double b = 0;
        for (int q = 0; q < n; ++q) {
            const FourierJob& J = jobs[i0 + q];
            const double io = (double)J.ft->nt * J.nc * ((forward ? in64 : out64) ? 8.0 : 4.0);
            const double hat = (double)J.ft->nf * J.ft->m2 * J.nc * (forward ? 4.0 : 4.0);
            b += io + hat + (!forward && J.yh ? 4.0 * J.ft->nt * J.nc : 0.0);
        }
        return b;
    };
    // launches of up to FT_JOBS consecutive jobs with the same sector count
    auto batches = [&]() {
        std::vector<std::pair<size_t, int>> b;
        for (size_t i0 = 0; i0 < jobs.size();) {
            int n = 1;
            while (i0 + n < jobs.size() && n < FT_JOBS && jobs[i0 + n].ft->nth == jobs[i0].ft->nth) ++n;
            b.push_back({i0, n});
            i0 += n;
        }
        return b;
    };
    auto set_tw = [&](DftArgs& a, int nth) {
        for (int k = 0; k < nth; ++k)
            a.tw[k] = make_float2((float)std::cos(TWO_PI * k / nth), (float)std::sin(TWO_PI * k / nth));
    };
    for (const auto& bt : batches()) {
        const size_t i0 = bt.first;
        DftArgs a;
        a.n = bt.second;
        for (int q = 0; q < a.n; ++q) a.j[q] = dft_job(i0 + q, true);
        const int nth = jobs[i0].ft->nth;
        set_tw(a, nth);
        const double by = dft_bytes(i0, a.n, true);
        int nb = 0;
        for (int q = 0; q < a.n; ++q) nb = std::max(nb, a.j[q].nb);
        const dim3 gd(maxnc, a.n), bs(fdft_threads(nb));
        if (in64) {
            if (nth == 24) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<24, double>), gd, bs, dft_smem(24, nb), cx.st, a);
            else if (nth == 30) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<30, double>), gd, bs, dft_smem(30, nb), cx.st, a);
            else if (nth == 36) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<36, double>), gd, bs, dft_smem(36, nb), cx.st, a);
            else TIMED_LAUNCH("fourier_dft", 0.0, by, fdft_kernel<double>, gd, 192, 0, cx.st, a);
        } else {
            if (nth == 24) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<24, float>), gd, bs, dft_smem(24, nb), cx.st, a);
            else if (nth == 30) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<30, float>), gd, bs, dft_smem(30, nb), cx.st, a);
            else if (nth == 36) TIMED_LAUNCH("fourier_dft", 0.0, by, (fdft_rep<36, float>), gd, bs, dft_smem(36, nb), cx.st, a);
            else TIMED_LAUNCH("fourier_dft", 0.0, by, fdft_kernel<float>, gd, 192, 0, cx.st, a);
        }
    }
    // one GEMM of order 2 n3 per job and frequency: Y^_f = inv(C^_f) X^_f in real form
    std::vector<TcProblem> P;
    std::vector<TcOperands> O;
    for (size_t k = 0; k < jobs.size(); ++k) {
        const FourierTube& F = *jobs[k].ft;
        const int nc = jobs[k].nc;
        for (int f = 0; f < F.nf; ++f) {
            const size_t ao = (size_t)f * F.m2 * F.ldk, xo = (size_t)f * F.ldk * nc;
            TcProblem p;
            p.M = F.m2; p.N = nc; p.K = F.m2;
            p.alpha = 1.f; p.beta = 0.f;
            p.C = yh[k].get() + xo; p.c_rs = 1; p.c_cs = F.ldk;
            TcOperands o;
            o.A = {const_cast<bf16*>(F.Ah.get()) + ao, const_cast<bf16*>(F.Al.get()) + ao, F.m2, F.m2, F.ldk};
            o.B = {xh[k].get() + xo, xl[k].get() + xo, nc, F.m2, F.ldk};
            P.push_back(p);
            O.push_back(o);
        }
    }
    tc_gemm(P, O, cx.err, nullptr, cx.st);
    for (const auto& bt : batches()) {
        const size_t i0 = bt.first;
        DftArgs a;
        a.n = bt.second;
        for (int q = 0; q < a.n; ++q) a.j[q] = dft_job(i0 + q, false);
        const int nth = jobs[i0].ft->nth;
        set_tw(a, nth);
        const double by = dft_bytes(i0, a.n, false);
        int nb = 0;
        for (int q = 0; q < a.n; ++q) nb = std::max(nb, a.j[q].nb);
        const dim3 gs(maxnc, a.n), bs(idft_threads(nb));
        if (out64) {
            if (nth == 24) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<24, double>), gs, bs, dft_smem(24, nb), cx.st, a);
            else if (nth == 30) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<30, double>), gs, bs, dft_smem(30, nb), cx.st, a);
            else if (nth == 36) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<36, double>), gs, bs, dft_smem(36, nb), cx.st, a);
            else TIMED_LAUNCH("fourier_dft", 0.0, by, idft_kernel<double>, dim3(maxnc, a.n), 64, 0, cx.st, a);
        } else {
            if (nth == 24) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<24, float>), gs, bs, dft_smem(24, nb), cx.st, a);
            else if (nth == 30) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<30, float>), gs, bs, dft_smem(30, nb), cx.st, a);
            else if (nth == 36) TIMED_LAUNCH("fourier_dft", 0.0, by, (idft_rep<36, float>), gs, bs, dft_smem(36, nb), cx.st, a);
            else TIMED_LAUNCH("fourier_dft", 0.0, by, idft_kernel<float>, dim3(maxnc, a.n), 64, 0, cx.st, a);
        }
    }
}

}  // namespace sqbem
