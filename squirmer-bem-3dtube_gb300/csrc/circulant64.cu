// circulant64.cu -- see circulant64.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "assemble.cuh"
#include "circulant64.cuh"
#include "common.cuh"
#include "dense.cuh"
#include "tube_fourier.cuh"

namespace sqbem {

namespace {

constexpr double TWO_PI = 6.283185307179586476925286766559;
constexpr int MAXF = FT_MAX_SECTORS / 2 + 1;
constexpr int NEWTON_STEPS = 3;  // an FP32 inverse's 1e-4 .. 1e-3, squared three times

struct Twiddles {
    double2 t[FT_MAX_SECTORS];  // (cos, sin) of 2 pi k / nth
};
Twiddles twiddles(int nth) {
    Twiddles w;
    for (int k = 0; k < nth; ++k) w.t[k] = make_double2(std::cos(TWO_PI * k / nth), std::sin(TWO_PI * k / nth));
    return w;
}

// C^_f[r, (b, be)] = sum_d w^{f d} sum_g T0[r, 3 panel(b, d) + g] R_d[g][be], as the real
// form of every frequency and as FP32 complex.  Thread: row r; blockIdx.y: column.
__global__ void chat64_kernel(const double* __restrict__ T0, const int* __restrict__ panel, int nth, int nb, int nf,
                              const __grid_constant__ Twiddles tw, double* __restrict__ M, float2* __restrict__ C) {
    const int n3 = 3 * nb, m2 = 2 * n3;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n3) return;
    const int c = blockIdx.y, b = c / 3, be = c % 3;
    double re[MAXF], im[MAXF];
#pragma unroll
    for (int f = 0; f < MAXF; ++f) re[f] = im[f] = 0.0;
    for (int d = 0; d < nth; ++d) {
        const double* col = T0 + r + 3LL * panel[b * nth + d] * n3;
        const double cs = tw.t[d].x, sn = tw.t[d].y;
        const double v = be == 2 ? col[2LL * n3] : be == 0 ? cs * col[0] + sn * col[n3] : cs * col[n3] - sn * col[0];
        int k = 0;  // f d mod nth
#pragma unroll
        for (int f = 0; f < MAXF; ++f) {
            if (f < nf) {
                re[f] = fma(v, tw.t[k].x, re[f]);
                im[f] = fma(v, tw.t[k].y, im[f]);
                k += d;
                if (k >= nth) k -= nth;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < MAXF; ++f)
        if (f < nf) {
            double* const m = M + (long long)f * m2 * m2;
            m[r + (long long)c * m2] = re[f];
            m[n3 + r + (long long)(n3 + c) * m2] = re[f];
            m[n3 + r + (long long)c * m2] = im[f];
            m[r + (long long)(n3 + c) * m2] = -im[f];
            C[(long long)f * n3 * n3 + (long long)c * n3 + r] = make_float2((float)re[f], (float)im[f]);
        }
}

// X <- the real form of the FP32 complex inverse; blockIdx.y: column of the block, .z: frequency
__global__ void realform64_kernel(const float2* __restrict__ C, int n3, double* __restrict__ X) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y, m2 = 2 * n3;
    if (r >= n3) return;
    const float2 v = C[(long long)blockIdx.z * n3 * n3 + (long long)c * n3 + r];
    double* const m = X + (long long)blockIdx.z * m2 * m2;
    m[r + (long long)c * m2] = v.x;
    m[n3 + r + (long long)(n3 + c) * m2] = v.x;
    m[n3 + r + (long long)c * m2] = v.y;
    m[r + (long long)(n3 + c) * m2] = -v.y;
}

__global__ void identity_kernel(double* __restrict__ R, int m2) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r < m2) R[(long long)blockIdx.z * m2 * m2 + (long long)c * m2 + r] = r == c ? 1.0 : 0.0;
}

// Forward transform of one column per CTA: xh[f][j m2 + r] = (1 / nth) sum_s w^{-f s}
// (R_s^T x_panel(a, s))_al, r = (a, al), and + n3 for the imaginary part.  The sectors s and
// nth - s share a cosine and have opposite sines; for even nth so do s and nth / 2 - s up to
// (-1)^f.  The sums and differences are formed once in shared memory, which leaves
// nth / 4 FMAs each for the real and imaginary part of a frequency (the FP64 pipe is the
// bound; shared-memory traffic is not).
__global__ void __launch_bounds__(256) fdft64_kernel(const double* __restrict__ x, long long ldx,
                                                     const int* __restrict__ panel, int nth, int nb, int nf, int nc,
                                                     const __grid_constant__ Twiddles tw, double* __restrict__ xh,
                                                     int per) {
    extern __shared__ double sm[];
    __shared__ double2 tws[FT_MAX_SECTORS];
    // this CTA's representatives: per of them from a0 on, rows r0 .. of the column's transform
    const int a0 = blockIdx.y * per, r0 = 3 * a0, all3 = 3 * nb;
    nb = min(per, nb - a0);
    panel += a0 * nth;
    const int n3 = 3 * nb, ld = nth | 1, hn = nth / 2, j = blockIdx.x;
    const bool even = (nth & 1) == 0;
    if (threadIdx.x < nth) tws[threadIdx.x] = tw.t[threadIdx.x];
    x += j * ldx;
    for (int e = threadIdx.x; e < nb * nth; e += blockDim.x) {
        const int s = e % nth, a = e / nth;
        const double* xp = x + 3LL * panel[e];
        const double x0 = xp[0], x1 = xp[1], c = tw.t[s].x, sn = tw.t[s].y;
        double* v = sm + 3 * a * ld + s;
        v[0] = c * x0 + sn * x1;
        v[ld] = c * x1 - sn * x0;
        v[2 * ld] = xp[2];
    }
    __syncthreads();
    // s = 1 .. : v[s] = sum, v[nth - s] = difference
    const int np = (nth - 1) / 2;
    for (int e = threadIdx.x; e < n3 * np; e += blockDim.x) {
        double* v = sm + (e / np) * ld;
        const int s = 1 + e % np;
        const double a = v[s], b = v[nth - s];
        v[s] = a + b;
        v[nth - s] = a - b;
    }
    __syncthreads();
    // even nth: the same for s and nth / 2 - s: v[s] serves even f, v[nth / 2 - s] odd f
    const int nq = even ? (hn + 1) / 2 : 0;  // s = 0 .. nq - 1 with s < nth / 2 - s
    for (int e = threadIdx.x; e < n3 * nq; e += blockDim.x) {
        double* v = sm + (e / nq) * ld;
        const int s = e % nq;
        const double a = v[s], b = v[hn - s];
        v[s] = a + b;
        v[hn - s] = a - b;
        if (s > 0) {
            const double p = v[nth - s], q = v[hn + s];
            v[nth - s] = p - q;
            v[hn + s] = p + q;
        }
    }
    __syncthreads();
    const double scale = 1.0 / nth;
    for (int e = threadIdx.x; e < n3 * nf; e += blockDim.x) {
        const int f = e / n3, r = e - f * n3;
        const double* v = sm + r * ld;
        double re, im = 0.0;
        int k = 0;
        if (even) {
            const bool odd = f & 1;
            re = odd ? v[hn] : v[0];
            int s = 1;
            for (; 2 * s < hn; ++s) {
                k += f;
                if (k >= nth) k -= nth;
                re = fma(odd ? v[hn - s] : v[s], tws[k].x, re);
                im = fma(odd ? v[hn + s] : v[nth - s], -tws[k].y, im);
            }
            if (2 * s == hn) {
                k += f;
                if (k >= nth) k -= nth;
                re = fma(v[s], tws[k].x, re);
                im = fma(v[nth - s], -tws[k].y, im);
            }
        } else {
            re = v[0];
            for (int s = 1; s <= np; ++s) {
                k += f;
                if (k >= nth) k -= nth;
                re = fma(v[s], tws[k].x, re);
                im = fma(v[nth - s], -tws[k].y, im);
            }
        }
        double* o = xh + ((long long)f * nc + j) * 2 * all3 + r0 + r;
        o[0] = re * scale;
        o[all3] = im * scale;
    }
}

// Inverse transform of one column per CTA, with the same pairings: y~_s = sum over all
// frequencies of w^{f s} y^_f, y_panel(a, s) = R_s y~_s.
__global__ void __launch_bounds__(256) idft64_kernel(const double* __restrict__ yh, const int* __restrict__ panel,
                                                     int nth, int nb, int nf, int nc,
                                                     const __grid_constant__ Twiddles tw, double* __restrict__ y,
                                                     long long ldy, int per) {
    extern __shared__ double sm[];
    __shared__ double2 tws[FT_MAX_SECTORS];
    const int a0 = blockIdx.y * per, r0 = 3 * a0, all3 = 3 * nb;
    nb = min(per, nb - a0);
    panel += a0 * nth;
    const int n3 = 3 * nb, ld = nth | 1, lf = 2 * nf + 1, hn = nth / 2, j = blockIdx.x;
    const bool even = (nth & 1) == 0;
    double* const v = sm;             // n3 x ld: sectors
    double* const w = sm + n3 * ld;   // n3 x lf: (re, im) per frequency, weighted
    if (threadIdx.x < nth) tws[threadIdx.x] = tw.t[threadIdx.x];
    for (int e = threadIdx.x; e < n3 * nf; e += blockDim.x) {
        const int f = e / n3, r = e - f * n3;
        const double* o = yh + ((long long)f * nc + j) * 2 * all3 + r0 + r;
        const double g = f == 0 || 2 * f == nth ? 1.0 : 2.0;
        w[r * lf + 2 * f] = g * o[0];
        w[r * lf + 2 * f + 1] = g * o[all3];
    }
    __syncthreads();
    const int ns = even ? hn / 2 + 1 : hn + 1;  // s = 0 .. ns - 1
    for (int e = threadIdx.x; e < n3 * ns; e += blockDim.x) {
        const int s = e / n3, r = e - s * n3;
        const double* p = w + r * lf;
        double* o = v + r * ld;
        // cosine and sine sums over the even and the odd frequencies
        double ae = 0.0, be = 0.0, ao = 0.0, bo = 0.0;
        int k = 0;
        for (int f = 0; f < nf; f += 2) {
            ae = fma(tws[k].x, p[2 * f], ae);
            be = fma(tws[k].y, p[2 * f + 1], be);
            k += s;
            if (k >= nth) k -= nth;
            if (f + 1 < nf) {
                ao = fma(tws[k].x, p[2 * f + 2], ao);
                bo = fma(tws[k].y, p[2 * f + 3], bo);
                k += s;
                if (k >= nth) k -= nth;
            }
        }
        const double A = ae + ao, B = be + bo;
        o[s] = A - B;
        if (s > 0 && 2 * s != nth) o[nth - s] = A + B;
        if (even && 2 * s != hn) {  // sector nth / 2 - s: odd frequencies' cosines and even ones' sines change sign
            const double A2 = ae - ao, B2 = bo - be;
            o[hn - s] = A2 - B2;
            if (s > 0) o[hn + s] = A2 + B2;
        }
    }
    __syncthreads();
    y += j * ldy;
    for (int e = threadIdx.x; e < nb * nth; e += blockDim.x) {
        const int s = e % nth, a = e / nth;
        const double* q = v + 3 * a * ld + s;
        const double v0 = q[0], v1 = q[ld], c = tw.t[s].x, sn = tw.t[s].y;
        double* yp = y + 3LL * panel[e];
        yp[0] = c * v0 - sn * v1;
        yp[1] = sn * v0 + c * v1;
        yp[2] = q[2 * ld];
    }
}

size_t fdft_smem(int nth, int nb) { return sizeof(double) * 3 * nb * (nth | 1); }
size_t idft_smem(int nth, int nb) { return fdft_smem(nth, nb) + sizeof(double) * 3 * nb * (2 * (nth / 2 + 1) + 1); }
constexpr size_t SMEM_MAX = 200 * 1024;

__global__ void rule_tie_kernel(const double* __restrict__ tgt, int nT, const PanelRec* __restrict__ src, int nS,
                                int* flag) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (p >= nS) return;
    const double dx = src[p].c[0] - tgt[3 * i], dy = src[p].c[1] - tgt[3 * i + 1], dz = src[p].c[2] - tgt[3 * i + 2];
    const double d2 = dx * dx + dy * dy + dz * dz, h2 = src[p].h * src[p].h;
    bool tie = false;
    for (double t : {9.0, 2.25, 0.5625}) tie |= fabs(d2 - t * h2) <= 2e-11 * t * h2;
    if (tie) atomicOr(flag, 1);
}

__global__ void deflate_sector0_kernel(double* __restrict__ S, int n3, const int* __restrict__ rep_panel,
                                       const PanelRec* __restrict__ P, double sc) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r >= n3) return;
    const int q = c / 3;
    S[r + (long long)c * n3] += sc * P[rep_panel[r / 3]].n[r % 3] * P[q].n[c % 3] * P[q].area;
}

__global__ void fold_kernel(const double* __restrict__ T0, const int* __restrict__ panel, int nth, int nb,
                            const __grid_constant__ Twiddles tw, double* __restrict__ M) {
    const int n3 = 3 * nb, r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n3) return;
    const int c = blockIdx.y, b = c / 3, be = c % 3;
    double s = 0.0;
    for (int d = 0; d < nth; ++d) {
        const double* col = T0 + r + 3LL * panel[b * nth + d] * n3;
        const double cs = tw.t[d].x, sn = tw.t[d].y;
        s += be == 2 ? col[2LL * n3] : be == 0 ? cs * col[0] + sn * col[n3] : cs * col[n3] - sn * col[0];
    }
    M[r + (long long)c * n3] = s;
}

// max |R| as the bits of a non-negative double
__global__ void max_abs_bits_kernel(const double* __restrict__ R, size_t n, unsigned long long* out) {
    double m = 0.0;
    bool nan = false;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = fabs(R[i]);
        nan |= !(v <= 1.7e308);
        m = fmax(m, v);
    }
    unsigned long long b = nan ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
        b = t > b ? t : b;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(out, b);
}

void set_limits() {
    static std::once_flag once;
    std::call_once(once, [] {
        CUDA_CHECK(cudaFuncSetAttribute(fdft64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
        CUDA_CHECK(cudaFuncSetAttribute(idft64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
    });
}

bool switched_off(const char* name) {
    const char* e = std::getenv(name);
    return e && std::atoi(e) == 0;
}

}  // namespace

bool circulant64_supported(const TubeSymmetry& sym) {
    return fourier_supported(sym) && idft_smem(sym.nth, sym.nb) <= SMEM_MAX && !switched_off("SQBEM_TUBE_SYMMETRY") &&
           !switched_off("SQBEM_TUBE_FOURIER");
}

void assemble_sector0(const std::vector<PanelRec>& host, const PanelRec* dev, const TubeSymmetry& sym, double mu,
                      double* S, double* D, int* tie, cudaStream_t st) {
    const int nb = sym.nb, P = nb * sym.nth, n3 = 3 * nb;
    std::vector<double> hc(3 * (size_t)nb);
    for (int a = 0; a < nb; ++a)
        for (int k = 0; k < 3; ++k) hc[3 * a + k] = host[sym.rep_panel[a]].c[k];
    DevBuf<double> tc(hc.size(), st);
    tc.upload(hc.data(), hc.size());
    DevBuf<int> self(nb, st);
    self.upload(sym.rep_panel.data(), nb);
    BlockJob<double> j;
    j.tgt = tc.get();
    j.nT = nb;
    j.src = dev;
    j.nS = P;
    j.self_of = self.get();
    j.S = S;
    j.s_rs = 1;
    j.s_cs = n3;
    j.D = D;
    j.d_rs = 1;
    j.d_cs = n3;
    j.sscale = 1.0 / (EIGHT_PI * mu);
    j.dscale = -1.0 / EIGHT_PI;
    assemble_block(j, (int)std::min<long long>((long long)nb * P, 64LL << 20), st, false);
    LAUNCH(rule_tie_kernel, dim3(ceil_div(P, 128), nb), 128, 0, st, tc.get(), nb, dev, P, tie);
}

void deflate_sector0(double* S, const PanelRec* dev, const TubeSymmetry& sym, int P, double sc, cudaStream_t st) {
    DevBuf<int> rep(sym.nb, st);
    rep.upload(sym.rep_panel.data(), sym.nb);
    LAUNCH(deflate_sector0_kernel, dim3(ceil_div(3 * sym.nb, 64), 3 * P), 64, 0, st, S, 3 * sym.nb, rep.get(), dev, sc);
}

void fold_sector0(const double* T0, const int* panel, int nth, int nb, double* M, cudaStream_t st) {
    LAUNCH(fold_kernel, dim3(ceil_div(3 * nb, 64), 3 * nb), 64, 0, st, T0, panel, nth, nb, twiddles(nth), M);
}

bool Circulant64::build(const TubeSymmetry& sym, const double* T0, const int* tie, cudaStream_t st) {
    ready = false;
    nth = sym.nth;
    nb = sym.nb;
    nf = nth / 2 + 1;
    n3 = 3 * nb;
    m2 = 2 * n3;
    nt = n3 * nth;
    set_limits();
    panel.alloc(sym.panel.size(), st);
    panel.upload(sym.panel.data(), sym.panel.size());
    const size_t one = (size_t)m2 * m2, all = one * nf;
    DevBuf<double> C(all, st), R(all, st);
    DevBuf<float2> c32((size_t)nf * n3 * n3, st);
    inv.alloc(all, st);
    // [0]: Gauss-Jordan, [1]: a wait ran out, [2 .. 3]: the largest entry of the last residual
    DevBuf<int> flag(4, st);
    flag.zero();
    const dim3 gb(ceil_div(n3, 64), n3);
    LAUNCH(chat64_kernel, gb, 64, 0, st, T0, panel.get(), nth, nb, nf, twiddles(nth), C.get(), c32.get());
    gauss_jordan_blocks(c32.get(), nf, n3, flag.get(), st);
    LAUNCH(realform64_kernel, dim3(gb.x, gb.y, nf), 64, 0, st, c32.get(), n3, inv.get());
    OzMat a, x, r;
    a.split(C.get(), 1, m2, m2, m2, st, false, nf, one);
    for (int it = 0; it < NEWTON_STEPS; ++it) {
        LAUNCH(identity_kernel, dim3(ceil_div(m2, 128), m2, nf), 128, 0, st, R.get(), m2);
        x.split(inv.get(), m2, 1, m2, m2, st, true, nf, one);
        oz_gemm(a, x, -1.0, 1.0, R.get(), m2, flag.get() + 1, st, one);
        if (it + 1 == NEWTON_STEPS)
            LAUNCH(max_abs_bits_kernel, 152, 256, 0, st, R.get(), all,
                   reinterpret_cast<unsigned long long*>(flag.get() + 2));
        x.split(inv.get(), 1, m2, m2, m2, st, false, nf, one);
        r.split(R.get(), m2, 1, m2, m2, st, true, nf, one);
        oz_gemm(x, r, 1.0, 1.0, inv.get(), m2, flag.get() + 1, st, one);
    }
    digits.split(inv.get(), 1, m2, m2, m2, st, false, nf, one);
    int h[4], htie = 0;
    flag.download(h, 4);
    if (tie) {
        CUDA_CHECK(cudaMemcpyAsync(&htie, tie, sizeof(int), cudaMemcpyDeviceToHost, st));
        count_d2h(sizeof(int));
    }
    CUDA_CHECK(cudaStreamSynchronize(st));
    if (h[1]) fail(SQBEM_ERR_TIMEOUT, "Fourier blocks: a bounded wait in the FP64 tensor-core product expired");
    // the residual before the last step; the step squares it
    double res;
    static_assert(sizeof res == 2 * sizeof(int), "two words");
    std::memcpy(&res, h + 2, sizeof res);
    ready = !h[0] && !htie && res <= 1e-9;
    if (!ready) {
        inv.release();
        digits = OzMat();
    }
    return ready;
}

void Circulant64::solve(double* B, long long ldb, int nrhs, cudaStream_t st, int* err, bool transpose) const {
    if (nrhs <= 0) return;
    // few columns at a time through the FP64 pipe; many through the digits (of the inverses,
    // not of their transposes)
    if (nrhs > SK_N && (nrhs < 64 || transpose || !err)) {
        for (int c = 0; c < nrhs; c += SK_N) solve(B + c * ldb, ldb, std::min(SK_N, nrhs - c), st, err, transpose);
        return;
    }
    const Twiddles tw = twiddles(nth);
    const long long one = (long long)m2 * m2, plane = (long long)m2 * nrhs;
    // a CTA per column, or, for few columns, per 4 representatives of one (their transforms are
    // independent): one column on one SM took 100 us
    const int per = nrhs < 304 ? 4 : nb;
    const dim3 grid(nrhs, ceil_div(nb, per));
    DevBuf<double> xh((size_t)nf * plane, st);
    TIMED_LAUNCH("fourier_dft", 0.0, 8.0 * nrhs * (nt + (double)nf * m2), fdft64_kernel, grid, 256, fdft_smem(nth, per), st,
                 B, ldb, panel.get(), nth, nb, nf, nrhs, tw, xh.get(), per);
    if (nrhs <= SK_N) {
        DevBuf<double> yh((size_t)nf * plane, st);
        gemm64_few(transpose, m2, nrhs, m2, 1.0, inv.get(), m2, xh.get(), m2, 0.0, yh.get(), m2, st, nf, one, plane,
                   plane);
        xh = std::move(yh);
    } else {
        OzMat x;
        x.split(xh.get(), m2, 1, nrhs, m2, st, true, nf, plane);
        oz_gemm(digits, x, 1.0, 0.0, xh.get(), m2, err, st, plane);
    }
    TIMED_LAUNCH("fourier_dft", 0.0, 8.0 * nrhs * (nt + (double)nf * m2), idft64_kernel, grid, 256, idft_smem(nth, per), st,
                 xh.get(), panel.get(), nth, nb, nf, nrhs, tw, B, ldb, per);
}

}  // namespace sqbem
