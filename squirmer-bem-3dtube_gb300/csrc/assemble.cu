// assemble.cu -- panel-quadrature assembly of the BEM blocks, panel integrals
// and the field (representation formula) on the GPU.
//
// Physics, as in the reference (src/utils/kernels.hpp:8-21, 29-82):
//   SL_ij = int_p G_ij dS,  G_ij(r) = d_ij/|r| + r_i r_j/|r|^3,
//   DL_ij = int_p T_ijk m_k dS,  T_ijk(r) = -6 r_i r_j r_k/|r|^5,  r = x - x0,
// with the rule chosen by d = |c_p - x0| / h_p: d >= 3 -> 7 points, >= 1.5 ->
// 28, >= 0.75 -> 112, else 448 (Dunavant-7 on 1/4/16/64 sub-triangles), and the
// self panel by a Duffy transform over three sub-triangles with 10 x 10
// Gauss-Legendre points (DL = 0 there, since r.m = 0 on a flat panel).
//
// GPU structure (one block = a set of target centroids x sources panels):
//   far_kernel   one thread per (target, source) pair, 64 targets x 16 sources
//                per CTA; source panels staged in shared memory; pairs with
//                d >= 3 use the 7-point rule in registers and write their 3x3
//                blocks (coalesced: consecutive threads own consecutive rows of
//                a column-major block); pairs with d < 3 and the self pair are
//                appended to a near list.
//   near_kernel  one warp per near pair: the lanes split the 28/112/448 rule
//                points (or the 300 Duffy points), reduce with warp shuffles,
//                and lanes 0..8 write the entries.  Entries have fixed positions,
//                so the result does not depend on the list order.
//   rowsum / completion kernels: the completed double layer adds -sum_p D_ip to
//                the diagonal 3x3 blocks (duct_flow.hpp:103-105,
//                swimmer.hpp:218-220), computed by a fixed-order reduction over
//                the stored D block (deterministic).
// Precision: FP64 everywhere in SQBEM_FP64 mode.  In SQBEM_MIXED mode the
// relative vectors (vertex and centroid offsets) and the rule choice are FP64,
// rounded once; the far (7) and near (28/112) rules are evaluated in FP32 from
// them, while the 448-point near-singular rule and the Duffy self integrals stay
// FP64, with a reciprocal square root refined from an FP32 seed (rsqrt_nr).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <vector>

#include "assemble.cuh"
#include "bem/utils/quadrature.hpp"
#include "common.cuh"

namespace cg = cooperative_groups;

namespace sqbem {

// ---------------------------------------------------------------- tables
struct QPoint {
    double l0, l1, l2, w;
};
struct QPointF {
    float l0, l1, l2, w;
};
__host__ __device__ constexpr int rule_off(int r) { return r <= 0 ? 0 : r == 1 ? 7 : r == 2 ? 35 : r == 3 ? 147 : 595; }
__device__ QPoint d_rule[595];
__device__ QPointF d_rulef[595];
__constant__ QPoint c_rule7[7];
__constant__ QPointF c_rule7f[7];
__device__ double d_gl_x[10], d_gl_w[10];
__device__ QPoint d_duffy[100];  // (x_a, x_b, w_a * w_b) for the 10 x 10 GL grid

static std::once_flag g_table_once[64];

void init_tables() {
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) fail(SQBEM_ERR_ARG, "device ordinal %d out of range", dev);
    std::call_once(g_table_once[dev], [] {
        std::vector<QPoint> h;
        std::vector<QPointF> hf;
        for (const auto& R : bem::rules())
            for (size_t q = 0; q < R.W.size(); ++q) {
                h.push_back({R.L[q][0], R.L[q][1], R.L[q][2], R.W[q]});
                hf.push_back({(float)R.L[q][0], (float)R.L[q][1], (float)R.L[q][2], (float)R.W[q]});
            }
        if (h.size() != 595) fail(SQBEM_ERR_ARG, "quadrature table has %zu points", h.size());
        CUDA_CHECK(cudaMemcpyToSymbol(d_rule, h.data(), sizeof(QPoint) * 595));
        CUDA_CHECK(cudaMemcpyToSymbol(d_rulef, hf.data(), sizeof(QPointF) * 595));
        CUDA_CHECK(cudaMemcpyToSymbol(c_rule7, h.data(), sizeof(QPoint) * 7));
        CUDA_CHECK(cudaMemcpyToSymbol(c_rule7f, hf.data(), sizeof(QPointF) * 7));
        std::vector<double> gx, gw;
        bem::gauss_legendre01(10, gx, gw);
        CUDA_CHECK(cudaMemcpyToSymbol(d_gl_x, gx.data(), sizeof(double) * 10));
        CUDA_CHECK(cudaMemcpyToSymbol(d_gl_w, gw.data(), sizeof(double) * 10));
        std::vector<QPoint> duf;
        for (int a = 0; a < 10; ++a)
            for (int b = 0; b < 10; ++b) duf.push_back({gx[a], gx[b], 0.0, gw[a] * gw[b]});
        CUDA_CHECK(cudaMemcpyToSymbol(d_duffy, duf.data(), sizeof(QPoint) * 100));
        CUDA_CHECK(cudaDeviceSynchronize());
    });
}

// ---------------------------------------------------------------- kernel sums
// Unique entries of the two symmetric 3x3 results plus the 1/|r| diagonal term.
template <class T>
struct Acc {
    T dg, sxx, sxy, sxz, syy, syz, szz, dxx, dxy, dxz, dyy, dyz, dzz;
    __device__ void zero() { dg = sxx = sxy = sxz = syy = syz = szz = dxx = dxy = dxz = dyy = dyz = dzz = T(0); }
};

// 1/sqrt(x) in FP64 for the mixed path's near-singular and self integrals: the
// FP32 seed y0 = rsqrtf(x) (relative error e0 below ~2^-21.5, including the
// rounding of x to FP32) refined by one Newton step for f(y) = 1/y^2 - x,
// y1 = y0 (3 - x y0^2) / 2, whose relative error is 1.5 e0^2 + O(e0^3) < 1e-13.
// Four FP64 operations instead of a full-precision FP64 reciprocal square root.
// x is a squared distance between quadrature point and target, far inside the
// FP32 range (and never 0: the Duffy and Gauss points are interior).
__device__ __forceinline__ double rsqrt_nr(double x) {
    const double y = (double)rsqrtf((float)x);
    return y * fma(-0.5 * x * y, y, 1.5);
}

template <bool NR>
__device__ __forceinline__ double rsqrt_t(double x) {
    if constexpr (NR) return rsqrt_nr(x);
    else return rsqrt(x);
}
template <bool NR>
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }

// One quadrature node: accumulate w G(r) and w T(r).m (kernels.hpp:29-40).
// NR: FP64 with rsqrt_nr (the mixed path's FP64 integrals).
template <class T, bool WITH_DL, bool NR = false>
__device__ __forceinline__ void accum(Acc<T>& A, T rx, T ry, T rz, T w, T mx, T my, T mz) {
    const T r2 = rx * rx + ry * ry + rz * rz;
    const T ir = rsqrt_t<NR>(r2);
    const T ir2 = ir * ir;
    const T ir3 = ir * ir2;
    const T s = w * ir3;
    A.dg += w * ir;
    const T sx = s * rx, sy = s * ry, sz = s * rz;
    A.sxx += sx * rx; A.sxy += sx * ry; A.sxz += sx * rz;
    A.syy += sy * ry; A.syz += sy * rz; A.szz += sz * rz;
    if (WITH_DL) {
        const T d = T(-6) * w * (rx * mx + ry * my + rz * mz) * ir3 * ir2;
        const T dx = d * rx, dy = d * ry, dz = d * rz;
        A.dxx += dx * rx; A.dxy += dx * ry; A.dxz += dx * rz;
        A.dyy += dy * ry; A.dyz += dy * rz; A.dzz += dz * rz;
    }
}

template <class T>
__device__ __forceinline__ void warp_reduce(Acc<T>& A) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        A.dg += __shfl_xor_sync(0xffffffffu, A.dg, o);
        A.sxx += __shfl_xor_sync(0xffffffffu, A.sxx, o);
        A.sxy += __shfl_xor_sync(0xffffffffu, A.sxy, o);
        A.sxz += __shfl_xor_sync(0xffffffffu, A.sxz, o);
        A.syy += __shfl_xor_sync(0xffffffffu, A.syy, o);
        A.syz += __shfl_xor_sync(0xffffffffu, A.syz, o);
        A.szz += __shfl_xor_sync(0xffffffffu, A.szz, o);
        A.dxx += __shfl_xor_sync(0xffffffffu, A.dxx, o);
        A.dxy += __shfl_xor_sync(0xffffffffu, A.dxy, o);
        A.dxz += __shfl_xor_sync(0xffffffffu, A.dxz, o);
        A.dyy += __shfl_xor_sync(0xffffffffu, A.dyy, o);
        A.dyz += __shfl_xor_sync(0xffffffffu, A.dyz, o);
        A.dzz += __shfl_xor_sync(0xffffffffu, A.dzz, o);
    }
}

// entry (a, b) of SL or DL from the accumulator
template <class T>
__device__ __forceinline__ T sl_entry(const Acc<T>& A, int a, int b) {
    const int k = a * 3 + b;
    T v = k == 0 ? A.sxx : k == 1 || k == 3 ? A.sxy : k == 2 || k == 6 ? A.sxz
        : k == 4 ? A.syy : k == 5 || k == 7 ? A.syz : A.szz;
    return a == b ? v + A.dg : v;
}
template <class T>
__device__ __forceinline__ T dl_entry(const Acc<T>& A, int a, int b) {
    const int k = a * 3 + b;
    return k == 0 ? A.dxx : k == 1 || k == 3 ? A.dxy : k == 2 || k == 6 ? A.dxz
         : k == 4 ? A.dyy : k == 5 || k == 7 ? A.dyz : A.dzz;
}

// Rule index of kernels.hpp:74-75 evaluated exactly as the reference does:
// d = |c - x0| / h with round-to-nearest products and sums in the reference's
// order (no FMA contraction), IEEE sqrt and division -- so a pair sitting on a
// threshold picks the same rule.
__device__ __forceinline__ int rule_of(const PanelRec& P, double x, double y, double z) {
    const double dx = P.c[0] - x, dy = P.c[1] - y, dz = P.c[2] - z;
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const double d = __ddiv_rn(__dsqrt_rn(d2), P.h);
    return d < 0.75 ? 3 : (d < 1.5 ? 2 : (d < 3.0 ? 1 : 0));
}

// ---------------------------------------------------------------- whole-pair integrals
// Sum over one rule's points split across the 32 lanes of a warp (after the
// call every lane holds the complete sums).  FP64 or FP32 evaluation from the
// FP64 relative vertex vectors e_k = V_k - x0.
template <class T, bool NR = false>
__device__ void warp_rule(Acc<T>& A, const PanelRec& P, double x, double y, double z, int rule, int lane) {
    A.zero();
    const T e0x = (T)(P.v[0] - x), e0y = (T)(P.v[1] - y), e0z = (T)(P.v[2] - z);
    const T e1x = (T)(P.v[3] - x), e1y = (T)(P.v[4] - y), e1z = (T)(P.v[5] - z);
    const T e2x = (T)(P.v[6] - x), e2y = (T)(P.v[7] - y), e2z = (T)(P.v[8] - z);
    const T mx = (T)P.n[0], my = (T)P.n[1], mz = (T)P.n[2];
    const T area = (T)P.area;
    const int q0 = rule_off(rule), q1 = rule_off(rule + 1);
    for (int q = q0 + lane; q < q1; q += 32) {
        T l0, l1, l2, w;
        if constexpr (sizeof(T) == 8) {
            const QPoint Q = d_rule[q];
            l0 = Q.l0; l1 = Q.l1; l2 = Q.l2; w = Q.w;
        } else {
            const QPointF Q = d_rulef[q];
            l0 = Q.l0; l1 = Q.l1; l2 = Q.l2; w = Q.w;
        }
        const T rx = l0 * e0x + l1 * e1x + l2 * e2x;
        const T ry = l0 * e0y + l1 * e1y + l2 * e2y;
        const T rz = l0 * e0z + l1 * e1z + l2 * e2z;
        accum<T, true, NR>(A, rx, ry, rz, w * area, mx, my, mz);
    }
    warp_reduce(A);
}

// The FP64 sums of a rule for the FP64 mode, v[0 .. 5] = sum w rr/|r|^3, v[6 .. 11] = sum w
// rr/|r|^5, v[12] = sum w/|r| over this lane's points: r.m is the same at every point of a
// flat panel and, with the area, enters once per entry.  (It comes from a vertex here, from a node
// in the far kernels: the centroid lies off the plane by its own rounding, which grows with the
// distance from the origin of the coordinates.)
__device__ __forceinline__ void lane_rule64(double (&v)[16], const PanelRec& P, double x, double y, double z, int rule,
                                            int lane) {
    const double e0x = P.v[0] - x, e0y = P.v[1] - y, e0z = P.v[2] - z;
    const double e1x = P.v[3] - x, e1y = P.v[4] - y, e1z = P.v[5] - z;
    const double e2x = P.v[6] - x, e2y = P.v[7] - y, e2z = P.v[8] - z;
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = 0.0;
    const int q1 = rule_off(rule + 1);
    for (int q = rule_off(rule) + lane; q < q1; q += 32) {
        const QPoint Q = d_rule[q];
        const double rx = Q.l0 * e0x + Q.l1 * e1x + Q.l2 * e2x;
        const double ry = Q.l0 * e0y + Q.l1 * e1y + Q.l2 * e2y;
        const double rz = Q.l0 * e0z + Q.l1 * e1z + Q.l2 * e2z;
        const double ir = rsqrt(rx * rx + ry * ry + rz * rz), ir2 = ir * ir, t = Q.w * ir, a3 = t * ir2, a5 = a3 * ir2;
        const double rr[6] = {rx * rx, rx * ry, rx * rz, ry * ry, ry * rz, rz * rz};
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            v[k] = fma(a3, rr[k], v[k]);
            v[6 + k] = fma(a5, rr[k], v[6 + k]);
        }
        v[12] += t;
    }
}
// Warp sums of 16 values by halving: lane l ends with value l & 15 (15 + 1 FP64 additions
// instead of 5 per value).
__device__ __forceinline__ double warp_sum16(double (&v)[16], int lane) {
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1)
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const bool up = lane & h;
            const double give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// FP32 evaluation of a 7/28/112-point rule from centroid-relative offsets:
// r = (c - x0) + sum_k l_k (V_k - c).  The FP64 differences and their FP32
// roundings are spread over lanes 0..15 (one value each) and broadcast by
// shuffles, so a pair costs a few FP64 warp instructions instead of a dozen
// per lane (GB300's FP64 pipe runs at about 1/64 of the FP32 rate).
__device__ void warp_rule_f32(Acc<float>& A, const PanelRec* Pg, double x, double y, double z, int rule, int lane) {
    A.zero();
    // minuend: v (9), c, n, area (words 0 .. 8, 12 .. 14, 9 .. 11, 15 of the record);
    // subtrahend: c, x0, 0: one FP64 subtraction and one conversion for the warp
    const double* const w = reinterpret_cast<const double*>(Pg);
    const double hi = w[lane < 9 ? lane : lane < 12 ? lane + 3 : lane < 15 ? lane - 3 : 15];
    const double lo = lane < 9 ? w[12 + lane % 3] : lane == 9 ? x : lane == 10 ? y : lane == 11 ? z : 0.0;
    const float val = (float)(hi - lo);
    float d[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) d[k] = __shfl_sync(0xffffffffu, val, k);
    const float bx = __shfl_sync(0xffffffffu, val, 9), by = __shfl_sync(0xffffffffu, val, 10),
                bz = __shfl_sync(0xffffffffu, val, 11);
    const float mx = __shfl_sync(0xffffffffu, val, 12), my = __shfl_sync(0xffffffffu, val, 13),
                mz = __shfl_sync(0xffffffffu, val, 14), area = __shfl_sync(0xffffffffu, val, 15);
    const int q0 = rule_off(rule), q1 = rule_off(rule + 1);
    for (int q = q0 + lane; q < q1; q += 32) {
        const QPointF Q = d_rulef[q];
        const float rx = bx + (Q.l0 * d[0] + Q.l1 * d[3] + Q.l2 * d[6]);
        const float ry = by + (Q.l0 * d[1] + Q.l1 * d[4] + Q.l2 * d[7]);
        const float rz = bz + (Q.l0 * d[2] + Q.l1 * d[5] + Q.l2 * d[8]);
        accum<float, true>(A, rx, ry, rz, Q.w * area, mx, my, mz);
    }
    warp_reduce(A);
}

// Duffy self integral (kernels.hpp:50-65): x0 inside the panel; three
// sub-triangles (x0, V_e, V_e+1), x = x0 + u[(1 - v) e1 + v e2], Jacobian u J.
// The edge vectors and J are formed once per sub-triangle; the lanes split its
// 10 x 10 points.
template <bool NR = false>
__device__ void warp_self(Acc<double>& A, const PanelRec& P, double x, double y, double z, int lane) {
    A.zero();
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int f = e == 2 ? 0 : e + 1;
        const double e1x = P.v[3 * e] - x, e1y = P.v[3 * e + 1] - y, e1z = P.v[3 * e + 2] - z;
        const double e2x = P.v[3 * f] - x, e2y = P.v[3 * f + 1] - y, e2z = P.v[3 * f + 2] - z;
        const double cx = e1y * e2z - e1z * e2y, cy = e1z * e2x - e1x * e2z, cz = e1x * e2y - e1y * e2x;
        const double J = sqrt(cx * cx + cy * cy + cz * cz);
        for (int g = lane; g < 100; g += 32) {
            const QPoint Q = d_duffy[g];
            const double u = Q.l0, v = Q.l1;
            const double rx = u * ((1 - v) * e1x + v * e2x);
            const double ry = u * ((1 - v) * e1y + v * e2y);
            const double rz = u * ((1 - v) * e1z + v * e2z);
            accum<double, false, NR>(A, rx, ry, rz, Q.w * u * J, 0.0, 0.0, 0.0);
        }
    }
    warp_reduce(A);
}

// ---------------------------------------------------------------- near-pair list
// One list of capacity near_cap: the heavy pairs (448-point rule, self
// integral) fill it from the front, the light ones (28/112 points) from the back,
// so the near kernel can take the heavy ones first.  near_count[0], [1]: the
// heavy and light counts; [2]: the near kernel's work counter.  A slot is
// written only while it is inside the list; counts whose sum exceeds the
// capacity mean overflow (the near kernel then does nothing and the host
// fails the call).
template <class TO>
__device__ __forceinline__ void near_append(const BlockJob<TO>& job, int i, int p, int rule) {
    const bool heavy = rule >= 3;
    const int slot = atomicAdd(job.near_count + (heavy ? 0 : 1), 1);
    if (slot < job.near_cap) job.near_list[heavy ? slot : job.near_cap - 1 - slot] = make_int2(i, p | (rule << 28));
}

// ---------------------------------------------------------------- far kernel
constexpr int FAR_TGT = 64;   // targets per CTA (threads)
constexpr int FAR_SRC = 16;   // source panels per CTA

// FP64 mode: one thread per target.  The FP64 pipe (one warp instruction per 64 cycles and SM
// quarter) bounds it, so the CTA stages what depends on the source panel alone -- the 7 nodes'
// offsets from the centroid, 9 h^2 -- and a pair takes (c - x0) + o_q per node, r.m once (the
// panel is flat), the signs and the area once per entry, and a rule test without square
// root or division unless it lies within 1e-12 of the threshold or below: 270 FP64
// operations a pair instead of 400 (1392 x 1280 panels both ways and 1280 x 1280: 4.0 ms before).
constexpr int FAR64_WORDS = 30;
template <class TO, int SRC>
__global__ void __launch_bounds__(FAR_TGT) far_kernel(BlockJob<TO> job) {
    __shared__ double sp[SRC][FAR64_WORDS];  // o (21), c, n, 9 h^2, S scale, D scale
    const int p0 = blockIdx.y * SRC;
    const int ns = min(SRC, job.nS - p0);
    for (int e = threadIdx.x; e < ns * 10; e += FAR_TGT) {
        const int s = e / 10, q = e - 10 * s;
        const PanelRec& P = job.src[p0 + s];
        double* d = sp[s];
        if (q < 7) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                d[3 * q + k] = c_rule7[q].l0 * (P.v[k] - P.c[k]) + c_rule7[q].l1 * (P.v[3 + k] - P.c[k]) +
                               c_rule7[q].l2 * (P.v[6 + k] - P.c[k]);
        } else if (q == 7) {
            for (int k = 0; k < 3; ++k) d[21 + k] = P.c[k];
        } else if (q == 8) {
            for (int k = 0; k < 3; ++k) d[24 + k] = P.n[k];
        } else {
            d[27] = 9.0 * P.h * P.h * (1.0 + 1e-12);
            d[28] = P.area * job.sscale;
            d[29] = -6.0 * P.area * job.dscale;
        }
    }
    __syncthreads();
    const int i = blockIdx.x * FAR_TGT + threadIdx.x;
    if (i >= job.nT) return;
    const int self_p = job.same_mesh ? i : (job.self_of ? job.self_of[i] : -1);
    const double x = job.tgt[3 * i], y = job.tgt[3 * i + 1], z = job.tgt[3 * i + 2];
    for (int s = 0; s < ns; ++s) {
        const double* d = sp[s];
        const int p = p0 + s;
        const double bx = d[21] - x, by = d[22] - y, bz = d[23] - z;
        int rule = p == self_p ? 4 : 0;
        if (rule == 0 && !(bx * bx + by * by + bz * bz > d[27])) rule = rule_of(job.src[p], x, y, z);
        if (rule != 0) {
            near_append(job, i, p, rule);
            if (job.rule_count) atomicAdd(job.rule_count + rule, 1);
            continue;
        }
        double dg = 0, sxx = 0, sxy = 0, sxz = 0, syy = 0, syz = 0, szz = 0;
        double dxx = 0, dxy = 0, dxz = 0, dyy = 0, dyz = 0, dzz = 0;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const double rx = bx + d[3 * q], ry = by + d[3 * q + 1], rz = bz + d[3 * q + 2];
            const double ir = rsqrt(rx * rx + ry * ry + rz * rz), ir2 = ir * ir, t = c_rule7[q].w * ir;
            const double a3 = t * ir2, a5 = a3 * ir2;
            dg += t;
            const double xx = rx * rx, xy = rx * ry, xz = rx * rz, yy = ry * ry, yz = ry * rz, zz = rz * rz;
            sxx = fma(a3, xx, sxx); sxy = fma(a3, xy, sxy); sxz = fma(a3, xz, sxz);
            syy = fma(a3, yy, syy); syz = fma(a3, yz, syz); szz = fma(a3, zz, szz);
            if (job.D) {
                dxx = fma(a5, xx, dxx); dxy = fma(a5, xy, dxy); dxz = fma(a5, xz, dxz);
                dyy = fma(a5, yy, dyy); dyz = fma(a5, yz, dyz); dzz = fma(a5, zz, dzz);
            }
        }
        const long long r0 = 3LL * i, c0 = 3LL * p;
        auto put = [&](TO* o, long long rs, long long cs, double f, double xx, double xy, double xz, double yy, double yz,
                       double zz) {
            TO* e = o + r0 * rs + c0 * cs;
            const TO vxy = (TO)(f * xy), vxz = (TO)(f * xz), vyz = (TO)(f * yz);
            e[0] = (TO)(f * xx); e[rs] = vxy; e[2 * rs] = vxz;
            e[cs] = vxy; e[cs + rs] = (TO)(f * yy); e[cs + 2 * rs] = vyz;
            e[2 * cs] = vxz; e[2 * cs + rs] = vyz; e[2 * cs + 2 * rs] = (TO)(f * zz);
        };
        if (job.S) put(job.S, job.s_rs, job.s_cs, d[28], sxx + dg, sxy, sxz, syy + dg, syz, szz + dg);
        if (job.D)
            put(job.D, job.d_rs, job.d_cs, d[29] * ((bx + d[0]) * d[24] + (by + d[1]) * d[25] + (bz + d[2]) * d[26]), dxx,
                dxy, dxz, dyy, dyz, dzz);
    }
}

// FP32 view of a source panel for the mixed far field, formed once per block by
// far_prep_kernel: the offsets of the 7 quadrature nodes from the centroid
// (sum_k l_k (V_k - c), formed in FP64 and rounded once), the node weights of
// the single layer (w area) and of the double layer (-6 w area), the normal,
// the centroid as an unevaluated sum hi + lo of two floats, and the squared rule
// thresholds (0.75 h)^2, (1.5 h)^2, (3 h)^2 lowered (thlo) and raised (thhi) by
// 1e-5.  Everything here depends on the source panel only, so the pair loop
// forms a node as (c - x0) + o_q.
struct __align__(16) FarF {
    float o[21];
    float ws[7], wd[7];
    float n[3];
    float chi[3], clo[3];
    float thlo[3], thhi[3];
    float pad[2];
};
static_assert(sizeof(FarF) % 16 == 0, "FarF is copied as float4");

// v = hi + lo with hi = fl32(v) and lo = fl32(v - hi): the pair carries v to
// about 2^-48 relative, so a difference of two such pairs formed in FP32,
// (a_hi - b_hi) + (a_lo - b_lo), is within ~2.5 FP32 ulps of the exact one.
__device__ __forceinline__ void split2(double v, float& hi, float& lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

// FarF of every source panel and the hi + lo split (x, y, z hi; x, y, z lo) of
// every target: the only FP64 work of the mixed far field.
__device__ __forceinline__ void far_prep(const PanelRec* __restrict__ src, int nS, const double* __restrict__ tgt,
                                         int nT, FarF* __restrict__ srcf, float* __restrict__ tgtf, int k) {
    if (k < nS) {
        const PanelRec& P = src[k];
        FarF F;
        double d[9];
        for (int q = 0; q < 9; ++q) d[q] = P.v[q] - P.c[q % 3];
        for (int q = 0; q < 7; ++q) {
            const QPoint& R = c_rule7[q];
            for (int x = 0; x < 3; ++x) F.o[3 * q + x] = (float)(R.l0 * d[x] + R.l1 * d[3 + x] + R.l2 * d[6 + x]);
            F.ws[q] = (float)(R.w * P.area);
            F.wd[q] = (float)(-6.0 * R.w * P.area);
        }
        for (int q = 0; q < 3; ++q) {
            F.n[q] = (float)P.n[q];
            split2(P.c[q], F.chi[q], F.clo[q]);
        }
        const double h2 = P.h * P.h;
        const double t[3] = {0.5625 * h2, 2.25 * h2, 9.0 * h2};
        for (int q = 0; q < 3; ++q) {
            F.thlo[q] = (float)(t[q] * (1.0 - 1e-5));
            F.thhi[q] = (float)(t[q] * (1.0 + 1e-5));
        }
        F.pad[0] = F.pad[1] = 0.f;
        srcf[k] = F;
    }
    if (k < nT)
        for (int q = 0; q < 3; ++q) split2(tgt[3 * k + q], tgtf[6 * k + q], tgtf[6 * k + 3 + q]);
}

__global__ void far_prep_kernel(const PanelRec* __restrict__ src, int nS, const double* __restrict__ tgt, int nT,
                                FarF* __restrict__ srcf, float* __restrict__ tgtf) {
    far_prep(src, nS, tgt, nT, srcf, tgtf, blockIdx.x * blockDim.x + threadIdx.x);
}

// blockIdx.y: one of several panel sets or target sets
constexpr int PREP_MAX = 96;
struct PrepArgs {
    struct {
        const PanelRec* src;
        const double* tgt;
        FarF* srcf;
        float* tgtf;
        int nS, nT;
    } j[PREP_MAX];
};
__global__ void far_prep_group(const __grid_constant__ PrepArgs g) {
    const auto& j = g.j[blockIdx.y];
    far_prep(j.src, j.nS, j.tgt, j.nT, j.srcf, j.tgtf, blockIdx.x * blockDim.x + threadIdx.x);
}

// Mixed mode: as far_kernel, all in FP32.  c - x0 comes from the hi + lo pairs
// (relative error <= ~2.5 ulp per component, so d2 is within ~5e-7 of the exact
// value), and the rule from comparing d2 with the thresholds' 1e-5 bands: a
// pair clear of every band has the rule the reference's FP64 test gives; a
// pair inside a band (rare) takes the reference's exact test (rule_of).  The
// near kernel takes the rule from the list.  Near pairs are gathered in a
// shared-memory list first (heavy from the front, light from the back) and
// appended to the global list with one atomic per class at the end of the CTA,
// so no thread waits on a global atomic inside the pair loop.
// SRC: source panels per CTA (FAR_SRC, or fewer for blocks with few targets,
// such as the tube's sector-0 rows, so that the grid still fills the GPU).
// tag goes into the upper bits of a near entry's target (the job of a grouped launch).
template <class TO, int SRC>
__device__ __forceinline__ void far_f32(const BlockJob<TO>& job, const FarF* __restrict__ srcf,
                                        const float* __restrict__ tgtf, int tag) {
    constexpr int FAR_PAIRS = FAR_TGT * SRC;
    __shared__ FarF sf[SRC];
    __shared__ int2 nl[FAR_PAIRS];
    __shared__ int ncount[2], nbase[2], rcount[5];
    const int p0 = blockIdx.y * SRC;
    const int ns = min(SRC, job.nS - p0);
    {
        const float4* s4 = reinterpret_cast<const float4*>(srcf + p0);
        float4* d4 = reinterpret_cast<float4*>(sf);
        const int n4 = ns * (int)(sizeof(FarF) / sizeof(float4));
        for (int k = threadIdx.x; k < n4; k += blockDim.x) d4[k] = s4[k];
    }
    if (threadIdx.x < 2) ncount[threadIdx.x] = 0;
    if (threadIdx.x < 5) rcount[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * FAR_TGT + threadIdx.x;
    const int nsi = i < job.nT ? ns : 0;  // targets past the end take part in the barriers only
    float xh = 0.f, yh = 0.f, zh = 0.f, xl = 0.f, yl = 0.f, zl = 0.f;
    int self_p = -1;
    if (nsi > 0) {
        xh = tgtf[6 * i]; yh = tgtf[6 * i + 1]; zh = tgtf[6 * i + 2];
        xl = tgtf[6 * i + 3]; yl = tgtf[6 * i + 4]; zl = tgtf[6 * i + 5];
        self_p = job.same_mesh ? i : (job.self_of ? job.self_of[i] : -1);
    }
    const float ss = (float)job.sscale, ds = (float)job.dscale;
    // column-major outputs (row stride 1, every block of the mixed path): per
    // target row 3 i the row bases, per pair one column offset
    const bool colmajor = (!job.S || job.s_rs == 1) && (!job.D || job.d_rs == 1);
    const long long scs = job.s_cs, dcs = job.d_cs;
    TO* const Sr = job.S ? job.S + 3LL * i : nullptr;
    TO* const Dr = job.D ? job.D + 3LL * i : nullptr;
    for (int s = 0; s < nsi; ++s) {
        const FarF& F = sf[s];
        const int p = p0 + s;
        const float bx = (F.chi[0] - xh) + (F.clo[0] - xl);
        const float by = (F.chi[1] - yh) + (F.clo[1] - yl);
        const float bz = (F.chi[2] - zh) + (F.clo[2] - zl);
        const float d2 = bx * bx + by * by + bz * bz;
        int rule;
        if (p == self_p) rule = 4;
        else if (d2 > F.thhi[2]) rule = 0;
        else if (d2 < F.thlo[2] && d2 > F.thhi[1]) rule = 1;
        else if (d2 < F.thlo[1] && d2 > F.thhi[0]) rule = 2;
        else if (d2 < F.thlo[0]) rule = 3;
        else rule = rule_of(job.src[p], job.tgt[3 * i], job.tgt[3 * i + 1], job.tgt[3 * i + 2]);
        if (rule != 0) {
            const bool heavy = rule >= 3;
            const int slot = atomicAdd(&ncount[heavy ? 0 : 1], 1);  // at most FAR_PAIRS in total
            nl[heavy ? slot : FAR_PAIRS - 1 - slot] = make_int2(i | tag, p | (rule << 28));
            if (job.rule_count) atomicAdd(&rcount[rule], 1);
            continue;
        }
        Acc<float> A;
        A.zero();
        // r = (c - x0) + o_q; the accumulation of accum<float, true> with the
        // node weights precomputed
        const float mx = F.n[0], my = F.n[1], mz = F.n[2];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float rx = bx + F.o[3 * q], ry = by + F.o[3 * q + 1], rz = bz + F.o[3 * q + 2];
            const float r2 = rx * rx + ry * ry + rz * rz;
            const float ir = rsqrtf(r2);
            const float ir2 = ir * ir;
            const float ir3 = ir * ir2;
            const float sw = F.ws[q] * ir3;
            A.dg += F.ws[q] * ir;
            const float sx = sw * rx, sy = sw * ry, sz = sw * rz;
            A.sxx += sx * rx; A.sxy += sx * ry; A.sxz += sx * rz;
            A.syy += sy * ry; A.syz += sy * rz; A.szz += sz * rz;
            const float dd = (F.wd[q] * ir3) * ((rx * mx + ry * my + rz * mz) * ir2);
            const float dx = dd * rx, dy = dd * ry, dz = dd * rz;
            A.dxx += dx * rx; A.dxy += dx * ry; A.dxz += dx * rz;
            A.dyy += dy * ry; A.dyz += dy * rz; A.dzz += dz * rz;
        }
        if (colmajor) {
            // the 3x3 block at base + 3 p ld + a + b ld: one base per pair, the
            // columns b = 1, 2 at the hoisted strides, rows a as immediates
            if (Sr) {
                TO* sp = Sr + 3LL * p * scs;
#pragma unroll
                for (int b = 0; b < 3; ++b)
#pragma unroll
                    for (int a = 0; a < 3; ++a) sp[a + b * scs] = (TO)(sl_entry(A, a, b) * ss);
            }
            if (Dr) {
                TO* dp = Dr + 3LL * p * dcs;
#pragma unroll
                for (int b = 0; b < 3; ++b)
#pragma unroll
                    for (int a = 0; a < 3; ++a) dp[a + b * dcs] = (TO)(dl_entry(A, a, b) * ds);
            }
            continue;
        }
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const long long r = 3LL * i + a, c = 3LL * p + b;
                if (job.S) job.S[r * job.s_rs + c * job.s_cs] = (TO)(sl_entry(A, a, b) * ss);
                if (job.D) job.D[r * job.d_rs + c * job.d_cs] = (TO)(dl_entry(A, a, b) * ds);
            }
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        const int n = ncount[threadIdx.x];
        nbase[threadIdx.x] = n > 0 ? atomicAdd(job.near_count + threadIdx.x, n) : 0;
    }
    if (job.rule_count && threadIdx.x >= 1 && threadIdx.x < 5 && rcount[threadIdx.x] > 0)
        atomicAdd(job.rule_count + threadIdx.x, rcount[threadIdx.x]);
    __syncthreads();
    const int nh = ncount[0], nlt = ncount[1], cap = job.near_cap;
    for (int e = threadIdx.x; e < nh; e += FAR_TGT) {
        const int slot = nbase[0] + e;
        if (slot < cap) job.near_list[slot] = nl[e];
    }
    for (int e = threadIdx.x; e < nlt; e += FAR_TGT) {
        const int slot = nbase[1] + e;
        if (slot < cap) job.near_list[cap - 1 - slot] = nl[FAR_PAIRS - 1 - e];
    }
}

template <class TO, int SRC>
__global__ void __launch_bounds__(FAR_TGT, 8) far_kernel_f32(BlockJob<TO> job, const FarF* __restrict__ srcf,
                                                          const float* __restrict__ tgtf) {
    far_f32<TO, SRC>(job, srcf, tgtf, 0);
}

// Several blocks of one kind (every swimmer's tube rows, or sphere rows) per launch,
// blockIdx.z the block.  One by one a 1248 x 320 block took 9.5 us to prepare, 12.5 us for
// its 1600 short CTAs and 6.7 us for its near pairs, most of it launch and tail.
constexpr int GROUP_MAX = 48;
constexpr int TAG_SHIFT = 24;  // near entries: target below, block above
struct GroupArgs {
    int n;
    BlockJob<float> job[GROUP_MAX];
    const FarF* srcf[GROUP_MAX];
    const float* tgtf[GROUP_MAX];
};

template <int SRC>
__global__ void __launch_bounds__(FAR_TGT, 8) far_group_kernel(const __grid_constant__ GroupArgs g) {
    const BlockJob<float>& job = g.job[blockIdx.z];
    if ((int)(blockIdx.x * FAR_TGT) >= job.nT || (int)(blockIdx.y * SRC) >= job.nS) return;
    far_f32<float, SRC>(job, g.srcf[blockIdx.z], g.tgtf[blockIdx.z], (int)blockIdx.z << TAG_SHIFT);
}

// ---------------------------------------------------------------- near kernel
// Warps take pairs from a shared counter, heavy pairs first (a heavy pair costs
// up to 16x a light one; static striding left SMs idle for a third of the run).
// Each pair is computed whole by one warp, so the result does not depend on the
// order.
// list: the job that holds the near list; of(e): the job of a list entry.
template <class TO, bool MIXED, class Of>
__device__ __forceinline__ void near_pairs(const BlockJob<TO>& list, int imask, Of of) {
    const int lane = threadIdx.x & 31;
    const int nh = list.near_count[0], nl = list.near_count[1];
    if (nh + nl > list.near_cap) return;  // overflow: reported by the host
    // heavy pairs (448-point rule, self integrals) by warp index: warp g takes
    // g, g + W, ...; one-warp CTAs are dispatched round-robin over the SMs, so
    // consecutive heavy pairs run on different SMs' FP64 pipes (a shared counter
    // hands consecutive tickets to the warps of one SM).  Then the light pairs
    // from the counter.
    const int W = gridDim.x * (blockDim.x >> 5);
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int kh = gw;
    for (;;) {
        int k;
        if (kh < nh) {
            k = kh;
            kh += W;
        } else {
            int t = 0;
            if (lane == 0) t = atomicAdd(list.near_count + 2, 1);
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t >= nl) break;
            k = nh + t;
        }
        const int2 e = list.near_list[k < nh ? k : list.near_cap - 1 - (k - nh)];
        const BlockJob<TO>& job = of(e.x);
        const int i = e.x & imask, p = e.y & 0x0fffffff;
        const PanelRec P = job.src[p];
        const double x = job.tgt[3 * i], y = job.tgt[3 * i + 1], z = job.tgt[3 * i + 2];
        const int rule = e.y >> 28;  // exact rule (4 = self), decided by the far kernel
        double sl = 0, dl = 0;
        const int a = lane / 3, b = lane % 3;
        if (rule == 4) {
            Acc<double> A;
            warp_self<MIXED>(A, P, x, y, z, lane);
            if (lane < 9) { sl = sl_entry(A, a, b); dl = 0.0; }
        } else if (MIXED && rule < 3) {
            Acc<float> A;
            warp_rule_f32(A, job.src + p, x, y, z, rule, lane);
            if (lane < 9) { sl = sl_entry(A, a, b); dl = dl_entry(A, a, b); }
        } else if (MIXED) {
            Acc<double> A;
            warp_rule<double, MIXED>(A, P, x, y, z, rule, lane);
            if (lane < 9) { sl = sl_entry(A, a, b); dl = dl_entry(A, a, b); }
        } else {
            double v[16];
            lane_rule64(v, P, x, y, z, rule, lane);
            const double t = warp_sum16(v, lane);
            // entry (a, b): symmetric index into xx xy xz yy yz zz
            const int lo = min(a, b), hi = max(a, b), k = (lo == 0 ? 0 : lo == 1 ? 2 : 3) + hi;
            const double dg = __shfl_sync(0xffffffffu, t, 12);
            sl = __shfl_sync(0xffffffffu, t, k & 31);
            dl = __shfl_sync(0xffffffffu, t, (6 + k) & 31);
            if (a == b) sl += dg;
            sl *= P.area;
            dl *= -6.0 * P.area * ((P.v[0] - x) * P.n[0] + (P.v[1] - y) * P.n[1] + (P.v[2] - z) * P.n[2]);
        }
        if (lane < 9) {
            const long long r = 3LL * i + a, c = 3LL * p + b;
            if (job.S) job.S[r * job.s_rs + c * job.s_cs] = (TO)(sl * job.sscale);
            if (job.D) job.D[r * job.d_rs + c * job.d_cs] = (TO)(dl * job.dscale);
        }
    }
}

template <class TO, bool MIXED>
__global__ void __launch_bounds__(32, 24) near_kernel(BlockJob<TO> job) {
    near_pairs<TO, MIXED>(job, 0x7fffffff, [&](int) -> const BlockJob<TO>& { return job; });
}

__global__ void __launch_bounds__(32, 24) near_group_kernel(const __grid_constant__ GroupArgs g) {
    near_pairs<float, true>(g.job[0], (1 << TAG_SHIFT) - 1,
                            [&](int x) -> const BlockJob<float>& { return g.job[x >> TAG_SHIFT]; });
}

// 24 one-warp CTAs per SM (80 registers per thread): consecutive pairs of the list -- the heavy
// 448-point and self pairs come first -- go to warps of different SMs, so they do not queue
// on a few SMs' FP64 pipes
static int near_warps() {
    static int sms = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        int dev = 0;
        CUDA_CHECK(cudaGetDevice(&dev));
        CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    });
    return sms * 24;
}

template <class TO>
void assemble_block(const BlockJob<TO>& job0, int near_cap, cudaStream_t st, bool mixed) {
    if (job0.nT <= 0 || job0.nS <= 0) return;
    init_tables();
    BlockJob<TO> job = job0;
    DevBuf<int2> list((size_t)near_cap, st);
    DevBuf<int> count(3, st);
    count.zero();
    job.near_list = list.get();
    job.near_count = count.get();
    job.near_cap = near_cap;
    DevBuf<int> rc;
    if (kstats_on()) {
        rc.alloc(5, st);
        rc.zero();
        job.rule_count = rc.get();
    }
    dim3 grid(ceil_div(job.nT, FAR_TGT), ceil_div(job.nS, FAR_SRC));
    // few target blocks (the tube's sector-0 rows): 4 sources per CTA, 4x the CTAs
    const bool narrow = mixed && (long long)grid.x * grid.y < 2LL * 152 * 4;
    const dim3 grid4(grid.x, ceil_div(job.nS, 4));
    // credited work: every pair considered, at the 7-point rule; bytes written
    const double pairs = (double)job.nT * job.nS;
    const double fl = pairs * 7.0 * FLOPS_PER_EVAL;
    const double by = pairs * 9.0 * sizeof(TO) * ((job.S ? 1 : 0) + (job.D ? 1 : 0));
    if (mixed) {
        DevBuf<FarF> srcf((size_t)job.nS, st);
        DevBuf<float> tgtf((size_t)job.nT * 6, st);
        LAUNCH(far_prep_kernel, ceil_div(std::max(job.nS, job.nT), 128), 128, 0, st, job.src, job.nS, job.tgt, job.nT,
               srcf.get(), tgtf.get());
        if (narrow)
            TIMED_LAUNCH("assemble_far", fl, by, (far_kernel_f32<TO, 4>), grid4, FAR_TGT, 0, st, job, srcf.get(), tgtf.get());
        else
            TIMED_LAUNCH("assemble_far", fl, by, (far_kernel_f32<TO, FAR_SRC>), grid, FAR_TGT, 0, st, job, srcf.get(),
                         tgtf.get());
    } else {
        // a pair takes a warp 270 x 64 cycles, so 16 sources one after the other are 140 us: fewer
        // per CTA until every SM quarter has a warp (80 x 80 panels: 168 us with 16)
        const long long ctas = (long long)grid.x * grid.y;
        if (ctas >= 304) TIMED_LAUNCH("assemble_far", fl, by, (far_kernel<TO, FAR_SRC>), grid, FAR_TGT, 0, st, job);
        else if (ctas >= 76)
            TIMED_LAUNCH("assemble_far", fl, by, (far_kernel<TO, 4>), dim3(grid.x, ceil_div(job.nS, 4)), FAR_TGT, 0, st,
                         job);
        else
            TIMED_LAUNCH("assemble_far", fl, by, (far_kernel<TO, 1>), dim3(grid.x, job.nS), FAR_TGT, 0, st, job);
    }
    const int warps = near_warps();
    // credited FP64-pipe work of the near kernel (kernel statistics only, which
    // count the pairs per rule on the device): the 448-point rule and the self
    // integral, plus in FP64 mode the 28- and 112-point rules (FP32 in mixed mode)
    if (kstats_on()) {
        int* counts = kstat_pinned_ints(5);
        CUDA_CHECK(cudaMemcpyAsync(counts, rc.get(), 5 * sizeof(int), cudaMemcpyDeviceToHost, st));
        const double w[5] = {0.0, mixed ? 0.0 : 28.0 * FLOPS_PER_EVAL, mixed ? 0.0 : 112.0 * FLOPS_PER_EVAL,
                             448.0 * FLOPS_PER_EVAL, 300.0 * FLOPS_PER_EVAL_SL};
        char note[96];
        std::snprintf(note, sizeof note, "nT=%d nS=%d same=%d mixed=%d", job.nT, job.nS, job.same_mesh, (int)mixed);
        kstat_note(note);
        const int ks = kstat_begin(st);
        if (mixed) LAUNCH((near_kernel<TO, true>), warps, 32, 0, st, job);
        else LAUNCH((near_kernel<TO, false>), warps, 32, 0, st, job);
        kstat_end_counted(ks, "assemble_near", st, counts, w, 5, 0.0);
    } else if (mixed) {
        LAUNCH((near_kernel<TO, true>), warps, 32, 0, st, job);
    } else {
        LAUNCH((near_kernel<TO, false>), warps, 32, 0, st, job);
    }
    if ((long long)job.nT * job.nS > near_cap) {
        // the list could overflow only for blocks larger than its capacity
        int h[3] = {};
        count.download(h, 3);
        CUDA_CHECK(cudaStreamSynchronize(st));
        if ((long long)h[0] + h[1] > near_cap)
            fail(SQBEM_ERR_ARG, "near-pair list overflow (%lld > %d)", (long long)h[0] + h[1], near_cap);
    }
}

// FP32 blocks of the mixed path, column-major, by grouped launches.  Panel sets and target sets
// that several blocks share (the tube of an ensemble) are prepared once.  The near list of
// a launch holds every pair of its blocks, so it cannot overflow: launches of up to
// GROUP_MAX blocks and 32 M pairs.
void assemble_group(const std::vector<BlockJob<float>>& jobs, cudaStream_t st) {
    init_tables();
    for (size_t i0 = 0; i0 < jobs.size();) {
        GroupArgs g;
        PrepArgs pr;
        long long pairs = 0;
        int mt = 0, ms = 0, mp = 0, np = 0;
        std::vector<size_t> so, to;  // offsets into the prepared arrays
        size_t ns = 0, nt = 0;
        g.n = 0;
        while (i0 < jobs.size() && g.n < GROUP_MAX) {
            const BlockJob<float>& J = jobs[i0];
            if (J.nT <= 0 || J.nS <= 0) {
                ++i0;
                continue;
            }
            const long long p = (long long)J.nT * J.nS;
            if (J.nT >= 1 << TAG_SHIFT || p > 32LL << 20) {  // outside the group's forms
                if (g.n > 0) break;
                assemble_block(J, (int)std::min<long long>(p, 64LL << 20), st, true);
                ++i0;
                continue;
            }
            if (g.n > 0 && pairs + p > 32LL << 20) break;
            pairs += p;
            // this block's panel set and target set, or an earlier block's
            size_t a = ns, b = nt;
            for (int k = 0; k < g.n; ++k) {
                if (g.job[k].src == J.src && g.job[k].nS == J.nS) a = so[k];
                if (g.job[k].tgt == J.tgt && g.job[k].nT == J.nT) b = to[k];
            }
            const bool newS = a == ns, newT = b == nt;
            if (newS || newT) {
                pr.j[np].src = J.src;
                pr.j[np].tgt = J.tgt;
                pr.j[np].nS = newS ? J.nS : 0;
                pr.j[np].nT = newT ? J.nT : 0;
                pr.j[np].srcf = reinterpret_cast<FarF*>(a);
                pr.j[np].tgtf = reinterpret_cast<float*>(b);
                mp = std::max({mp, pr.j[np].nS, pr.j[np].nT});
                ++np;
            }
            so.push_back(a);
            to.push_back(b);
            if (newS) ns += J.nS;
            if (newT) nt += J.nT;
            g.job[g.n++] = J;
            mt = std::max(mt, J.nT);
            ms = std::max(ms, J.nS);
            ++i0;
        }
        if (g.n == 0) continue;
        DevBuf<FarF> srcf(ns, st);
        DevBuf<float> tgtf(6 * nt, st);
        DevBuf<int2> list((size_t)pairs, st);
        DevBuf<int> count(3, st), rc;
        count.zero();
        if (kstats_on()) {
            rc.alloc(5, st);
            rc.zero();
        }
        for (int k = 0; k < np; ++k) {
            pr.j[k].srcf = srcf.get() + reinterpret_cast<size_t>(pr.j[k].srcf);
            pr.j[k].tgtf = tgtf.get() + 6 * reinterpret_cast<size_t>(pr.j[k].tgtf);
        }
        for (int k = 0; k < g.n; ++k) {
            g.srcf[k] = srcf.get() + so[k];
            g.tgtf[k] = tgtf.get() + 6 * to[k];
            g.job[k].near_list = list.get();
            g.job[k].near_count = count.get();
            g.job[k].near_cap = (int)pairs;
            g.job[k].rule_count = rc.get();
        }
        double by = 0;
        for (int k = 0; k < g.n; ++k)
            by += 36.0 * g.job[k].nT * g.job[k].nS * ((g.job[k].S ? 1 : 0) + (g.job[k].D ? 1 : 0));
        LAUNCH(far_prep_group, dim3(ceil_div(mp, 128), np), 128, 0, st, pr);
        const dim3 grid(ceil_div(mt, FAR_TGT), ceil_div(ms, FAR_SRC), g.n), grid4(grid.x, ceil_div(ms, 4), g.n);
        // few CTAs (a swimmer or two): 4 sources each, as for one block
        if ((long long)grid.x * grid.y * grid.z < 2LL * 152 * 4)
            TIMED_LAUNCH("assemble_far", 7.0 * FLOPS_PER_EVAL * pairs, by, far_group_kernel<4>, grid4, FAR_TGT, 0, st, g);
        else
            TIMED_LAUNCH("assemble_far", 7.0 * FLOPS_PER_EVAL * pairs, by, far_group_kernel<FAR_SRC>, grid, FAR_TGT, 0, st,
                         g);
        if (kstats_on()) {
            int* counts = kstat_pinned_ints(5);
            CUDA_CHECK(cudaMemcpyAsync(counts, rc.get(), 5 * sizeof(int), cudaMemcpyDeviceToHost, st));
            const double w[5] = {0.0, 0.0, 0.0, 448.0 * FLOPS_PER_EVAL, 300.0 * FLOPS_PER_EVAL_SL};
            const int ks = kstat_begin(st);
            LAUNCH(near_group_kernel, near_warps(), 32, 0, st, g);
            kstat_end_counted(ks, "assemble_near", st, counts, w, 5, 0.0);
        } else {
            LAUNCH(near_group_kernel, near_warps(), 32, 0, st, g);
        }
    }
}

template void assemble_block<double>(const BlockJob<double>&, int, cudaStream_t, bool);
template void assemble_block<float>(const BlockJob<float>&, int, cudaStream_t, bool);

// ---------------------------------------------------------------- row sums
// partial[chunk][row][b] = sum over source panels p in the chunk of D(row, 3p + b).
// FP64 blocks are summed in FP64.  FP32 blocks are summed in FP32 pairs: each
// entry enters through an error-free TwoSum (the rounding error of every
// addition kept in a second FP32 sum), so the chunk's (double)s + (double)c is
// accurate to about 2^-48 of the sum of magnitudes -- what an FP64 sum of the
// FP32 entries gives -- at 6 FP32 operations per entry instead of an FP64 add
// (1/64 of the FP32 rate on GB300, which made this kernel FP64-bound).
__device__ __forceinline__ void two_sum_f(float& s, float& c, float x) {
    const float t = __fadd_rn(s, x);
    const float z = __fsub_rn(t, s);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z)));
    s = t;
}

template <class T>
__device__ __forceinline__ void rowsum_chunk(const T* __restrict__ D, long long rs, long long cs, int nrows,
                                             int ncolpanels, int chunk, double* __restrict__ partial) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= nrows) return;
    const int c = blockIdx.y;
    const int p0 = c * chunk, p1 = min(ncolpanels, p0 + chunk);
    double* o = partial + ((long long)c * nrows + row) * 3;
    if constexpr (sizeof(T) == sizeof(float)) {
        float s[3] = {0.f, 0.f, 0.f}, e[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
        for (int p = p0; p < p1; ++p) {
            const long long base = row * rs + 3LL * p * cs;
            const float d0 = __ldg(D + base), d1 = __ldg(D + base + cs), d2 = __ldg(D + base + 2 * cs);
            two_sum_f(s[0], e[0], d0);
            two_sum_f(s[1], e[1], d1);
            two_sum_f(s[2], e[2], d2);
        }
        for (int b = 0; b < 3; ++b) o[b] = (double)s[b] + (double)e[b];
    } else {
        double s0 = 0, s1 = 0, s2 = 0;
        for (int p = p0; p < p1; ++p) {
            const long long base = row * rs + 3LL * p * cs;
            s0 += (double)D[base];
            s1 += (double)D[base + cs];
            s2 += (double)D[base + 2 * cs];
        }
        o[0] = s0; o[1] = s1; o[2] = s2;
    }
}

template <class T>
__global__ void rowsum_kernel(const T* __restrict__ D, long long rs, long long cs, int nrows, int ncolpanels,
                              int chunk, double* __restrict__ partial) {
    rowsum_chunk(D, rs, cs, nrows, ncolpanels, chunk, partial);
}

// Add the chunked row sums (fixed order) to out[row * 3 + b]; the loads of eight chunks at once
__device__ __forceinline__ void rowsum_add(const double* __restrict__ partial, int nchunk, int nrows,
                                           double* __restrict__ out) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= nrows) return;
    double s0 = 0, s1 = 0, s2 = 0;
#pragma unroll 8
    for (int c = 0; c < nchunk; ++c) {
        const double* o = partial + ((long long)c * nrows + row) * 3;
        s0 += o[0]; s1 += o[1]; s2 += o[2];
    }
    out[row * 3] += s0;
    out[row * 3 + 1] += s1;
    out[row * 3 + 2] += s2;
}

__global__ void rowsum_finish(const double* __restrict__ partial, int nchunk, int nrows, double* __restrict__ out) {
    rowsum_add(partial, nchunk, nrows, out);
}

template <class T>
void add_rowsums(const T* D, long long rs, long long cs, int nrows, int ncolpanels, double* out, cudaStream_t st) {
    if (nrows <= 0 || ncolpanels <= 0) return;
    const int chunk = 32;  // panels per CTA column: many CTAs, so the loads overlap
    const int nchunk = ceil_div(ncolpanels, chunk);
    DevBuf<double> part((size_t)nchunk * nrows * 3, st);
    LAUNCH(rowsum_kernel<T>, dim3(ceil_div(nrows, 128), nchunk), 128, 0, st, D, rs, cs, nrows, ncolpanels, chunk,
           part.get());
    LAUNCH(rowsum_finish, ceil_div(nrows, 128), 128, 0, st, part.get(), nchunk, nrows, out);
}
template void add_rowsums<double>(const double*, long long, long long, int, int, double*, cudaStream_t);
template void add_rowsums<float>(const float*, long long, long long, int, int, double*, cudaStream_t);

// The FP32 row sums and the diagonal completion of several blocks per launch (blockIdx.z / .y
// the block; the same chunks and order as above).
struct SumArgs {
    RowsumJob j[GROUP_MAX];
    double* partial[GROUP_MAX];
};
__global__ void rowsum_group_kernel(const __grid_constant__ SumArgs g, int chunk) {
    const RowsumJob& J = g.j[blockIdx.z];
    if ((int)(blockIdx.y * chunk) >= J.npanels) return;
    rowsum_chunk(J.D, 1, J.ld, J.nrows, J.npanels, chunk, g.partial[blockIdx.z]);
}
__global__ void rowsum_finish_group(const __grid_constant__ SumArgs g, int chunk) {
    const RowsumJob& J = g.j[blockIdx.y];
    rowsum_add(g.partial[blockIdx.y], (J.npanels + chunk - 1) / chunk, J.nrows, J.out);
}

void add_rowsums_group(const std::vector<RowsumJob>& jobs, cudaStream_t st) {
    const int chunk = 32;
    for (size_t i0 = 0; i0 < jobs.size(); i0 += GROUP_MAX) {
        SumArgs g;
        const int n = (int)std::min<size_t>(GROUP_MAX, jobs.size() - i0);
        size_t total = 0;
        int mr = 0, mc = 0;
        for (int k = 0; k < n; ++k) {
            g.j[k] = jobs[i0 + k];
            const int nc = ceil_div(g.j[k].npanels, chunk);
            total += (size_t)nc * g.j[k].nrows * 3;
            mr = std::max(mr, g.j[k].nrows);
            mc = std::max(mc, nc);
        }
        if (mr <= 0 || mc <= 0) continue;
        DevBuf<double> part(total, st);
        size_t off = 0;
        for (int k = 0; k < n; ++k) {
            g.partial[k] = part.get() + off;
            off += (size_t)ceil_div(g.j[k].npanels, chunk) * g.j[k].nrows * 3;
        }
        LAUNCH(rowsum_group_kernel, dim3(ceil_div(mr, 128), mc, n), 128, 0, st, g, chunk);
        LAUNCH(rowsum_finish_group, dim3(ceil_div(mr, 128), n), 128, 0, st, g, chunk);
    }
}

// A(3i+a, 3i+b) -= rsum[(3i+a)*3 + b] (+ ext * delta_ab) for columns b with
// colmask bit b of mask[i] set (all three when mask == nullptr).
template <class T>
__global__ void diag_complete_kernel(T* A, long long rs, long long cs, int n, const double* __restrict__ rsum,
                                     double ext, const unsigned char* __restrict__ mask) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * n) return;
    const int i = t / 9, a = (t % 9) / 3, b = t % 3;
    if (mask && !((mask[i] >> b) & 1)) return;
    const long long r = 3LL * i + a, c = 3LL * i + b;
    const double v = (double)A[r * rs + c * cs] - rsum[r * 3 + b] - (a == b ? ext : 0.0);
    A[r * rs + c * cs] = (T)v;
}

template <class T>
void diag_complete(T* A, long long rs, long long cs, int n, const double* rsum, double ext,
                   const unsigned char* mask, cudaStream_t st) {
    if (n <= 0) return;
    LAUNCH(diag_complete_kernel<T>, ceil_div(9LL * n, 256), 256, 0, st, A, rs, cs, n, rsum, ext, mask);
}
template void diag_complete<double>(double*, long long, long long, int, const double*, double,
                                    const unsigned char*, cudaStream_t);
template void diag_complete<float>(float*, long long, long long, int, const double*, double,
                                   const unsigned char*, cudaStream_t);

// ---------------------------------------------------------------- panel integrals (API)
__global__ void pairs_kernel(int n, const PanelRec* __restrict__ P, const double* __restrict__ x0,
                             const int* __restrict__ self, double* SL, double* DL) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= n) return;
    const PanelRec R = P[warp];
    const double x = x0[3 * warp], y = x0[3 * warp + 1], z = x0[3 * warp + 2];
    Acc<double> A;
    const bool is_self = self[warp] != 0;
    if (is_self) warp_self(A, R, x, y, z, lane);
    else warp_rule<double>(A, R, x, y, z, rule_of(R, x, y, z), lane);
    if (lane < 9) {
        const int a = lane / 3, b = lane % 3;
        SL[9 * warp + lane] = sl_entry(A, a, b);
        DL[9 * warp + lane] = is_self ? 0.0 : dl_entry(A, a, b);
    }
}

void panel_pairs(int n, const PanelRec* P, const double* x0, const int* self, double* SL, double* DL,
                 cudaStream_t st) {
    if (n <= 0) return;
    init_tables();
    LAUNCH(pairs_kernel, ceil_div(32LL * n, 256), 256, 0, st, n, P, x0, self, SL, DL);
}

// ---------------------------------------------------------------- field
// u_j(x0) = sum_p [SL_p,ij f_p,i / (8 pi mu) - DL_p,ij u_p,i / (8 pi)]  (field.hpp:18-34)
//
// The lanes of a warp take panels, a warp PPW points (so that a staged panel serves
// several), or, for few points, two, four or the eight warps of a CTA (and the CTAs of a
// cluster) one point.  Pass 1 applies the 7-point rule to far panels while near ones (d < 3) are
// collected, in panel order, in shared memory; in pass 2 the warp integrates each near
// panel, its lanes splitting the rule's points.  Fixed order, hence deterministic.
//
// What bounds it is the FP64 pipe (64 cycles a warp instruction), so each panel's share of
// a tile is prepared once in shared memory, and
//   FP64    a flat panel's r.m is the same at all its nodes, and the node sums are formed
//           contracted: sum_q w f / r and sum_q (..) r, 27 FP64 operations a node;
//   mixed   nothing per pair is FP64: the rule by the bands of far_kernel_f32, the vertex
//           offsets V - x0 from FP32 pairs (TwoDiff, rounded as the FP64 difference's
//           conversion is but for one in 10^7), the products with f and u as FP32 pairs
//           (Dot2) within a tile's common power of two.
// 18 k points x 1712 panels in mixed precision: 12.5 ms with FP64 offsets, rule tests and
// products per pair.
constexpr int FIELD_WARPS = 8;
constexpr int FIELD_NEAR_CAP = 256;
constexpr int FT32 = 47, FT64 = 35;  // words per staged panel (odd: lanes on different banks)

__device__ __forceinline__ void two_diff(float a, float b, float& s, float& e) {
    s = __fsub_rn(a, b);
    const float t = __fsub_rn(s, a);
    e = __fsub_rn(__fsub_rn(a, __fsub_rn(s, t)), __fadd_rn(b, t));
}
// (s, c) += a (bh + bl)
__device__ __forceinline__ void dot2_add(float& s, float& c, float a, float bh, float bl) {
    const float p = __fmul_rn(a, bh), e = __fmaf_rn(a, bh, -p);
    const float t = __fadd_rn(s, p), z = __fsub_rn(t, s);
    c = __fadd_rn(c, __fadd_rn(__fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z)), __fmaf_rn(a, bl, e)));
    s = t;
}

struct FieldPoint {
    double x, y, z, u[3];
    int near;
};

// A panel's far share of a point's velocity in mixed precision from the FP64 coordinates and values, for
// tiles with an infinity or a NaN among f and u, or with panels far apart; nonzero rule: not far.
// Not inlined: the pair loop, which the instruction cache does not hold, does without its code.
struct FarShare {
    int rule;
    double u[3];
};
__device__ __noinline__ FarShare far_share(const PanelRec* P, const double* f, const double* u, double sscale,
                                           double dscale, double x, double y, double z) {
    FarShare r;
    r.rule = rule_of(*P, x, y, z);
    r.u[0] = r.u[1] = r.u[2] = 0.0;
    if (r.rule != 0) return r;
    float e[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) e[k] = (float)(P->v[k] - (k % 3 == 0 ? x : k % 3 == 1 ? y : z));
    const float mx = (float)P->n[0], my = (float)P->n[1], mz = (float)P->n[2], area = (float)P->area;
    Acc<float> A;
    A.zero();
#pragma unroll 1
    for (int q = 0; q < 7; ++q) {
        const float l0 = c_rule7f[q].l0, l1 = c_rule7f[q].l1, l2 = c_rule7f[q].l2, w = c_rule7f[q].w;
        accum<float, true>(A, l0 * e[0] + l1 * e[3] + l2 * e[6], l0 * e[1] + l1 * e[4] + l2 * e[7],
                           l0 * e[2] + l1 * e[5] + l2 * e[8], w * area, mx, my, mz);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            r.u[j] += (double)sl_entry(A, i, j) * f[i] * sscale + (double)dl_entry(A, i, j) * u[i] * dscale;
    return r;
}

// The panel-independent state of a point and its far sum over the panels of a tile, for both
// arithmetics: stage() writes one panel's record, pair() returns the rule and adds the
// panel if it is far, flush() moves the tile's sum to FP64.
template <class TC>
struct FieldArith;

template <>
struct FieldArith<double> {
    static constexpr int WORDS = FT64;
    static __device__ int exponent(const FieldJob&, int) { return 0; }
    static __device__ bool stage(double* d, const FieldJob& job, int p, const double*, int) {
        const PanelRec P = job.panels[p];
        double v[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = P.v[k] - P.c[k % 3];
#pragma unroll
        for (int q = 0; q < 7; ++q)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                d[3 * q + k] = c_rule7[q].l0 * v[k] + c_rule7[q].l1 * v[3 + k] + c_rule7[q].l2 * v[6 + k];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[21 + k] = P.n[k];
            d[24 + k] = P.c[k];
            d[28 + k] = job.f[3 * p + k] * (job.sscale * P.area);
            d[31 + k] = job.u[3 * p + k] * (-6.0 * job.dscale * P.area);
        }
        d[27] = 9.0 * P.h * P.h * (1.0 + 1e-12);
        return false;
    }
    double a[3];
    __device__ void offset(int, double, double) {}
    __device__ void begin() { a[0] = a[1] = a[2] = 0.0; }
    __device__ int pair(const double* d, const FieldJob& job, int p, const FieldPoint& X) {
        const double bx = d[24] - X.x, by = d[25] - X.y, bz = d[26] - X.z;
        // within 1e-12 of the threshold and below: the exact test
        if (!(bx * bx + by * by + bz * bz > d[27])) {
            const int rule = rule_of(job.panels[p], X.x, X.y, X.z);
            if (rule != 0) return rule;
        }
        const double rm = (bx + d[0]) * d[21] + (by + d[1]) * d[22] + (bz + d[2]) * d[23];
        const double fx = d[28], fy = d[29], fz = d[30], gx = d[31] * rm, gy = d[32] * rm, gz = d[33] * rm;
        double al = 0.0;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const double rx = bx + d[3 * q], ry = by + d[3 * q + 1], rz = bz + d[3 * q + 2];
            const double ir = rsqrt(rx * rx + ry * ry + rz * rz), ir2 = ir * ir, t = c_rule7[q].w * ir;
            al += t;
            const double fr = rx * fx + ry * fy + rz * fz, gr = rx * gx + ry * gy + rz * gz;
            const double be = t * ir2 * fma(gr, ir2, fr);
            a[0] = fma(be, rx, a[0]);
            a[1] = fma(be, ry, a[1]);
            a[2] = fma(be, rz, a[2]);
        }
        a[0] = fma(al, fx, a[0]);
        a[1] = fma(al, fy, a[1]);
        a[2] = fma(al, fz, a[2]);
        return 0;
    }
    __device__ void flush(FieldPoint& X, double) const {
#pragma unroll
        for (int k = 0; k < 3; ++k) X.u[k] += a[k];
    }
};

template <>
struct FieldArith<float> {
    static constexpr int WORDS = FT32;
    // the largest biased exponent of f / (8 pi mu) and u / (8 pi) on a panel; 0x7ff: not finite
    static __device__ int exponent(const FieldJob& job, int p) {
        int m = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            m = max(m, __double2hiint(job.f[3 * p + k] * job.sscale) & 0x7ff00000);
            m = max(m, __double2hiint(job.u[3 * p + k] * job.dscale) & 0x7ff00000);
        }
        return m >> 20;
    }
    // lengths relative to the origin o; f and u over 2^(ex - 1023).  True if the panel lies so far
    // from o for its size that the pairs' 2^-48 would show beside FP32's rounding.
    static __device__ bool stage(float* d, const FieldJob& job, int p, const double* o, int ex) {
        const PanelRec P = job.panels[p];
        float ext = 0.f;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            split2(P.v[k] - o[k % 3], d[k], d[9 + k]);
            ext = fmaxf(ext, fabsf(d[k]));
        }
        const double h2 = P.h * P.h, sc = ex > 0 && ex < 0x7ff ? scalbn(1.0, 1023 - ex) : 1.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double t = (k == 0 ? 0.5625 : k == 1 ? 2.25 : 9.0) * h2;
            d[18 + k] = (float)P.n[k];
            split2(P.c[k] - o[k], d[22 + k], d[25 + k]);
            d[28 + k] = (float)(t * (1.0 - 1e-5));
            d[31 + k] = (float)(t * (1.0 + 1e-5));
            split2(job.f[3 * p + k] * job.sscale * sc, d[34 + k], d[37 + k]);
            split2(job.u[3 * p + k] * job.dscale * sc, d[40 + k], d[43 + k]);
        }
        d[21] = (float)P.area;
        return ext > 4e6f * (float)P.h;
    }
    float xh[3], xl[3], s[3], c[3];
    // component k of the point's offset from the origin
    __device__ void offset(int k, float hi, float lo) {
        xh[k] = hi;
        xl[k] = lo;
    }
    __device__ void begin() {
#pragma unroll
        for (int k = 0; k < 3; ++k) s[k] = c[k] = 0.f;
    }
    __device__ int pair(const float* d, const FieldJob& job, int p, const FieldPoint& X) {
        const float bx = (d[22] - xh[0]) + (d[25] - xl[0]), by = (d[23] - xh[1]) + (d[26] - xl[1]),
                    bz = (d[24] - xh[2]) + (d[27] - xl[2]);
        const float d2 = bx * bx + by * by + bz * bz;
        if (!(d2 > d[33])) {
            int rule;
            if (d2 < d[30] && d2 > d[32]) rule = 1;
            else if (d2 < d[29] && d2 > d[31]) rule = 2;
            else if (d2 < d[28]) rule = 3;
            else rule = rule_of(job.panels[p], X.x, X.y, X.z);
            if (rule != 0) return rule;
        }
        float e[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            float hi, lo;
            two_diff(d[k], xh[k % 3], hi, lo);
            e[k] = __fadd_rn(hi, __fadd_rn(lo, __fsub_rn(d[9 + k], xl[k % 3])));
        }
        Acc<float> A;
        A.zero();
        const float mx = d[18], my = d[19], mz = d[20], area = d[21];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float l0 = c_rule7f[q].l0, l1 = c_rule7f[q].l1, l2 = c_rule7f[q].l2, w = c_rule7f[q].w;
            accum<float, true>(A, l0 * e[0] + l1 * e[3] + l2 * e[6], l0 * e[1] + l1 * e[4] + l2 * e[7],
                               l0 * e[2] + l1 * e[5] + l2 * e[8], w * area, mx, my, mz);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                dot2_add(s[j], c[j], sl_entry(A, i, j), d[34 + i], d[37 + i]);
                dot2_add(s[j], c[j], dl_entry(A, i, j), d[40 + i], d[43 + i]);
            }
        return 0;
    }
    __device__ void flush(FieldPoint& X, double scale) const {
#pragma unroll
        for (int k = 0; k < 3; ++k) X.u[k] = fma((double)s[k] + (double)c[k], scale, X.u[k]);
    }
};

// One near panel of one point by a warp.  u: lanes 0 .. 2 hold the component of their
// number; t (mixed, 28 and 112 points): lane 3 i + j holds the sum of its (i, j) terms,
// collected once per point.
template <bool MIXED>
__device__ void field_near(const FieldJob& job, int p, int rule, const FieldPoint& X, int lane, double& u, double& t) {
    if (MIXED && rule < 3) {
        Acc<float> A;
        warp_rule_f32(A, job.panels + p, X.x, X.y, X.z, rule, lane);
        const int i = lane / 3, j = lane - 3 * i;
        if (lane < 9) {
            t = fma((double)sl_entry(A, i, j), job.f[3 * p + i] * job.sscale, t);
            t = fma((double)dl_entry(A, i, j), job.u[3 * p + i] * job.dscale, t);
        }
        return;
    }
    const PanelRec& P = job.panels[p];
    const double e0x = P.v[0] - X.x, e0y = P.v[1] - X.y, e0z = P.v[2] - X.z;
    const double e1x = P.v[3] - X.x, e1y = P.v[4] - X.y, e1z = P.v[5] - X.z;
    const double e2x = P.v[6] - X.x, e2y = P.v[7] - X.y, e2z = P.v[8] - X.z;
    const double rm = -6.0 * (e0x * P.n[0] + e0y * P.n[1] + e0z * P.n[2]);
    const double ss = job.sscale * P.area, ds = job.dscale * P.area * rm;
    const double fx = job.f[3 * p] * ss, fy = job.f[3 * p + 1] * ss, fz = job.f[3 * p + 2] * ss;
    const double gx = job.u[3 * p] * ds, gy = job.u[3 * p + 1] * ds, gz = job.u[3 * p + 2] * ds;
    double al = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0;
    const int q1 = rule_off(rule + 1);
    for (int q = rule_off(rule) + lane; q < q1; q += 32) {
        const QPoint Q = d_rule[q];
        const double rx = Q.l0 * e0x + Q.l1 * e1x + Q.l2 * e2x;
        const double ry = Q.l0 * e0y + Q.l1 * e1y + Q.l2 * e2y;
        const double rz = Q.l0 * e0z + Q.l1 * e1z + Q.l2 * e2z;
        const double ir = rsqrt(rx * rx + ry * ry + rz * rz), ir2 = ir * ir, t = Q.w * ir;
        al += t;
        const double be = t * ir2 * fma(rx * gx + ry * gy + rz * gz, ir2, rx * fx + ry * fy + rz * fz);
        a0 = fma(be, rx, a0);
        a1 = fma(be, ry, a1);
        a2 = fma(be, rz, a2);
    }
    a0 = fma(al, fx, a0);
    a1 = fma(al, fy, a1);
    a2 = fma(al, fz, a2);
    // three sums over the warp: lane groups 0, 1 mod 4 and 2 mod 4 end with one component each
    const double k0 = __shfl_xor_sync(0xffffffffu, a0, 1), k1 = __shfl_xor_sync(0xffffffffu, a1, 1),
                 k2 = __shfl_xor_sync(0xffffffffu, a2, 1);
    double v = (lane & 1) ? a1 + k1 : a0 + k0, w = a2 + k2;
    const double vw = __shfl_xor_sync(0xffffffffu, v, 2), ww = __shfl_xor_sync(0xffffffffu, w, 2);
    v = (lane & 2) ? w + ww : v + vw;  // lanes 0, 1, 2 (mod 4): components 0, 1, 2 (3: 2 again)
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    u += v;
}

// PPW points per warp, each warp all panels (G = 1); or G warps per point, the CTAs of a cluster one
// point together where G = 8.  They share the panels: the CTAs every cluster-size-th one, so that near
// panels, which are neighbours, go to all of them; the warps 32 at a time (a warp costs the same
// with one lane as with all) and then, in turn, the entries of all their near lists.
template <class TC, int PPW, int G>
__global__ void __launch_bounds__(FIELD_WARPS * 32, 2) field_kernel(FieldJob job) {
    constexpr bool SHARED = G > 1, ALL = G == FIELD_WARPS;
    static_assert(!SHARED || PPW == 1, "shared points have warps of their own");
    constexpr int TP = SHARED ? 256 : 128;  // panels per tile
    constexpr int W = FieldArith<TC>::WORDS;
    extern __shared__ __align__(16) unsigned char field_smem[];
    TC* const tile = reinterpret_cast<TC*>(field_smem);
    int* const lists = reinterpret_cast<int*>(tile + TP * W);
    __shared__ int tex, twide;
    __shared__ double part[FIELD_WARPS][3];
    __shared__ int pnear[FIELD_WARPS];
    __shared__ double clsum[3];
    __shared__ int clnear;
    cg::cluster_group cl = cg::this_cluster();
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int ncl = ALL ? (int)cl.num_blocks() : 1, rank = ALL ? (int)cl.block_rank() : 0;
    const int sub = wl % G;  // of the point's warps
    const int pt0 = ALL ? blockIdx.x / ncl : (blockIdx.x * FIELD_WARPS + wl) / G * PPW;
    FieldPoint X[PPW];
    FieldArith<TC> F[PPW];
#pragma unroll
    for (int k = 0; k < PPW; ++k) {
        const int pt = min(pt0 + k, job.npts - 1);
        X[k].x = job.pts[3 * pt];
        X[k].y = job.pts[3 * pt + 1];
        X[k].z = job.pts[3 * pt + 2];
        X[k].u[0] = X[k].u[1] = X[k].u[2] = 0.0;
        X[k].near = 0;
    }
    // lane 3 k + c: component c of point k, for the offsets from a tile's origin
    const double xc = lane < 3 * PPW ? job.pts[3LL * min(pt0 + lane / 3, job.npts - 1) + lane % 3] : 0.0;
    // the origin of the staged lengths: a vertex of the first panel (no point, which may be
    // anything, has a say in another's result), or the one point of the CTA
    const double* o;
    auto set_origin = [&](const double* v) {
        o = v;
        if (sizeof(TC) != 4) return;
        float hi, lo;
        split2(xc - o[lane % 3], hi, lo);
#pragma unroll
        for (int k = 0; k < PPW; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                F[k].offset(c, __shfl_sync(0xffffffffu, hi, 3 * k + c), __shfl_sync(0xffffffffu, lo, 3 * k + c));
    };
    set_origin(ALL ? job.pts + 3LL * pt0 : job.P > 0 ? job.panels[0].v : job.pts);
    int* const list = lists + wl * PPW * FIELD_NEAR_CAP;
    for (int base = 0; base < job.P; base += ncl * TP) {
        const int mine = base + (int)threadIdx.x * ncl + rank;
        const bool has = (int)threadIdx.x < TP && mine < job.P;
        __syncthreads();
        if (threadIdx.x == 0) tex = twide = 0;
        __syncthreads();
        if (sizeof(TC) == 4 && has) {
            const int e = FieldArith<TC>::exponent(job, mine);
            if (e) atomicMax(&tex, e);
        }
        __syncthreads();
        const int ex = tex;
        if (has && FieldArith<TC>::stage(tile + threadIdx.x * W, job, mine, o, ex)) twide = 1;
        __syncthreads();
        bool wide = !ALL && twide != 0;
        if (wide && o != job.panels[base].v) {  // too far from the origin: once more from its own first panel
            __syncthreads();
            if (threadIdx.x == 0) twide = 0;
            set_origin(job.panels[base].v);
            __syncthreads();
            if (has && FieldArith<TC>::stage(tile + threadIdx.x * W, job, mine, o, ex)) twide = 1;
            __syncthreads();
            wide = twide != 0;
        }
        const bool plain = sizeof(TC) == 4 && (wide || ex == 0x7ff);
#pragma unroll
        for (int k = 0; k < PPW; ++k) F[k].begin();
        auto append = [&](int k, int p, int rule) {
            const unsigned m = __ballot_sync(0xffffffffu, rule > 0);
            if (rule > 0) {
                const int slot = X[k].near + __popc(m & ((1u << lane) - 1));
                if (slot < FIELD_NEAR_CAP) list[k * FIELD_NEAR_CAP + slot] = p | (rule << 28);
            }
            X[k].near += __popc(m);
        };
        for (int s = sub * 32; !plain && s < TP && base + s * ncl + rank < job.P; s += 32 * G) {
            const int q = s + lane, p = base + q * ncl + rank;
#pragma unroll
            for (int k = 0; k < PPW; ++k) append(k, p, p < job.P ? F[k].pair(tile + q * W, job, p, X[k]) : 0);
        }
#pragma unroll 1
        for (int s = sub * 32; plain && s < TP && base + s * ncl + rank < job.P; s += 32 * G) {
            const int p = base + (s + lane) * ncl + rank;
#pragma unroll
            for (int k = 0; k < PPW; ++k) {
                FarShare r = {};
                if (p < job.P)
                    r = far_share(job.panels + p, job.f + 3 * p, job.u + 3 * p, job.sscale, job.dscale, X[k].x, X[k].y, X[k].z);
#pragma unroll
                for (int j = 0; j < 3; ++j) X[k].u[j] += r.u[j];
                append(k, p, r.rule);
            }
        }
        const double scale = ex > 0 && ex < 0x7ff ? scalbn(1.0, ex - 1023) : 1.0;
#pragma unroll
        for (int k = 0; k < PPW; ++k) F[k].flush(X[k], scale);
    }
    if (SHARED) {
        if (lane == 0) pnear[wl] = X[0].near;
        __syncthreads();
    } else {
        __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < PPW; ++k) {
        // the far part: warp sums (fixed butterfly order), component j to lane j
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) X[k].u[j] += __shfl_xor_sync(0xffffffffu, X[k].u[j], d);
        double u = lane == 0 ? X[k].u[0] : lane == 1 ? X[k].u[1] : X[k].u[2];
        double t = 0.0;
        auto near = [&](int e) { field_near<sizeof(TC) == 4>(job, e & 0x0fffffff, e >> 28, X[k], lane, u, t); };
        if (SHARED) {
            for (int w = 0, first = sub; pt0 < job.npts && w < G; ++w) {  // first: of this warp's in list w
                const int c = min(pnear[wl - sub + w], FIELD_NEAR_CAP);
                for (; first < c; first += G) near(lists[(wl - sub + w) * FIELD_NEAR_CAP + first]);
                first -= c;
            }
        } else if (pt0 + k < job.npts) {
            const int nn = min(X[k].near, FIELD_NEAR_CAP);
            for (int n = 0; n < nn; ++n) near(list[k * FIELD_NEAR_CAP + n]);
        }
        if (sizeof(TC) == 4) u += t + __shfl_down_sync(0xffffffffu, t, 3) + __shfl_down_sync(0xffffffffu, t, 6);
        if (!SHARED && pt0 + k < job.npts) {
            if (lane < 3) job.out[3 * (pt0 + k) + lane] = u;
            if (lane == 0 && X[k].near > FIELD_NEAR_CAP) atomicExch(job.overflow, 1);
        }
        if (SHARED && lane < 3) part[wl][lane] = u;
    }
    if (SHARED && !ALL) {
        __syncthreads();
        if (sub == 0 && lane < 4 && pt0 < job.npts) {
            double u = 0.0;
            int n = 0;
            for (int w = wl; w < wl + G; ++w) {
                if (lane < 3) u += part[w][lane];
                else n += pnear[w];
            }
            if (lane < 3) job.out[3 * pt0 + lane] = u;
            else if (n > FIELD_NEAR_CAP) atomicExch(job.overflow, 1);
        }
    }
    if (ALL) {
        __syncthreads();
        if (threadIdx.x < 3) {
            double u = 0.0;
            for (int w = 0; w < FIELD_WARPS; ++w) u += part[w][threadIdx.x];
            clsum[threadIdx.x] = u;
        }
        if (threadIdx.x == 3) {
            int n = 0;
            for (int w = 0; w < FIELD_WARPS; ++w) n += pnear[w];
            clnear = n;
        }
        cl.sync();
        if (rank == 0 && threadIdx.x < 4) {
            double u = 0.0;
            int n = 0;
            for (int c = 0; c < ncl; ++c) {
                if (threadIdx.x < 3) u += cl.map_shared_rank(clsum, c)[threadIdx.x];
                else n += *cl.map_shared_rank(&clnear, c);
            }
            if (threadIdx.x < 3) job.out[3 * pt0 + threadIdx.x] = u;
            else if (n > FIELD_NEAR_CAP) atomicExch(job.overflow, 1);
        }
        cl.sync();
    }
}

__global__ void rsqrt_nr_kernel(int n, const double* __restrict__ x, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = rsqrt_nr(x[i]);
}

void rsqrt_nr_eval(int n, const double* x, double* y, cudaStream_t st) {
    if (n > 0) LAUNCH(rsqrt_nr_kernel, ceil_div(n, 256), 256, 0, st, n, x, y);
}

namespace {
template <class TC, int PPW, int G>
void field_launch(const FieldJob& job, int cluster, cudaStream_t st) {
    constexpr int TP = G > 1 ? 256 : 128;
    constexpr size_t smem =
        sizeof(TC) * TP * FieldArith<TC>::WORDS + sizeof(int) * FIELD_WARPS * PPW * FIELD_NEAR_CAP;
    static std::once_flag once;
    std::call_once(once, [] {
        CUDA_CHECK(cudaFuncSetAttribute((const void*)field_kernel<TC, PPW, G>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    });
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at[1];
    c.gridDim = dim3((unsigned)ceil_div(job.npts, FIELD_WARPS / G * PPW) * cluster);
    c.blockDim = dim3(FIELD_WARPS * 32);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    CUDA_CHECK(cudaLaunchKernelEx(&c, field_kernel<TC, PPW, G>, job));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

// Four points per warp once every SM has its 32 points, one per warp once it has eight.  Below that
// fewer points per CTA, with more warps each: staging the panels costs a CTA as much as eight (mixed)
// points' far panels or one's (FP64), so four or two points share it while every SM has a CTA, and
// then one point's warps, or the CTAs of a cluster, share its near panels.  The lines follow the
// whole rounds of the 152 SMs; in FP64, where the near panels weigh more than the staging, two CTAs
// per point also fill the ends of such rounds (with few panels they have too little to share).
// Whole calls, us, points in the duct / far away from it (120 of them are the call's own):
//   1680 panels, 1200 points, mixed: 445 / 334 (a CTA per point: 967 / 818; one warp: 491 / 307)
//   1680 panels,  300 points, FP64: 535 / 387 (four CTAs per point: 661 / 540; one warp: 1447 / 940)
//     56 panels,  300 points, FP64: - / 121 (four CTAs per point, 32 panels of a tile to each: 307; a warp
//                                   per point and nothing staged: 142)
template <class TC>
void field_dispatch(const FieldJob& job, cudaStream_t st) {
    const int n = job.npts;
    const bool fp64 = sizeof(TC) == 8;
    if (n >= 152 * FIELD_WARPS * 4) field_launch<TC, 4, 1>(job, 1, st);
    else if (n >= 152 * FIELD_WARPS) field_launch<TC, 1, 1>(job, 1, st);
    else if (n <= 38) field_launch<TC, 1, 8>(job, 8, st);
    else if (n <= 76 || (n <= 114 && job.P >= 1024)) field_launch<TC, 1, 8>(job, 4, st);
    else if (n <= 152 || (fp64 && job.P >= 64 && (n <= 228 || (n > 304 && n <= 456)))) field_launch<TC, 1, 8>(job, 2, st);
    else if (n <= 304 || (fp64 && n > 608 && n <= 912)) field_launch<TC, 1, 4>(job, 1, st);
    else field_launch<TC, 1, 2>(job, 1, st);
}
}  // namespace

void field_eval(const FieldJob& job, cudaStream_t st) {
    if (job.npts <= 0) return;
    init_tables();
    if (job.mixed) field_dispatch<float>(job, st);
    else field_dispatch<double>(job, st);
}

}  // namespace sqbem

// ---------------------------------------------------------------- adjoint contraction
namespace sqbem {

constexpr int ADJ_TT = 32;   // targets per CTA (one per lane)
constexpr int ADJ_ST = 32;   // source panels per CTA (staged in shared memory)
constexpr int ADJ_W = 4;     // warps, each a quarter of the sources
constexpr int ADJ_OUT = 6 * ADJ_MAX_MODES * 3;
constexpr int ADJ_WORDS = 41;  // staged words per source

// Gradients with respect to r of  phi_G = lam.G(r).f = (lam.f)/|r| + (lam.r)(f.r)/|r|^3
//   grad phi_G = [lam (f.r) + f (lam.r) - (lam.f) r] / |r|^3 - 3 (lam.r)(f.r) r / |r|^5
// and of phi_T = lam.(T(r).m).v = -6 (r.m)(lam.r)(v.r) / |r|^5
//   grad phi_T = -6 [m (lam.r)(v.r) + lam (r.m)(v.r) + v (r.m)(lam.r)] / |r|^5
//                + 30 (r.m)(lam.r)(v.r) r / |r|^7
// (kernels.hpp:8-9 differentiated).  Both are lam.C(f, v) with a 3 x 3 matrix C that does not
// know the adjoint vector, and C is linear in a few moments of the quadrature nodes.  So a
// pair sums its nodes into the moments
//   p = sum w r/|r|^3, y = sum w r/|r|^5, W = sum w r r/|r|^5, Q = sum w r r r/|r|^5,
//   Z = sum w r r r/|r|^7
// (symmetric; the zz. entries of Q and Z follow from the traces p and y), forms C per
// solution, and a target's C is summed over its sources before it meets the six adjoint
// vectors: 625 FP64 operations a far pair where the gradient per node, adjoint vector
// and solution took 5000 (FP64-bound, 10.6 ms for 1392 x 320 panels both ways).
struct AdjMoments {
    double p[3], y[3], W[6], Q[7], Z[7];  // W: xx xy xz yy yz zz; Q, Z: xxx xxy xxz xyy xyz yyy yyz
    __device__ void zero() {
#pragma unroll
        for (int k = 0; k < 3; ++k) p[k] = y[k] = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) W[k] = 0.0;
#pragma unroll
        for (int k = 0; k < 7; ++k) Q[k] = Z[k] = 0.0;
    }
    __device__ void node(double rx, double ry, double rz, double w) {
        const double ir = rsqrt(rx * rx + ry * ry + rz * rz), ir2 = ir * ir;
        const double a3 = w * ir * ir2, a5 = a3 * ir2, a7 = a5 * ir2;
        const double xx = rx * rx, xy = rx * ry, xz = rx * rz, yy = ry * ry, yz = ry * rz;
        p[0] = fma(a3, rx, p[0]); p[1] = fma(a3, ry, p[1]); p[2] = fma(a3, rz, p[2]);
        y[0] = fma(a5, rx, y[0]); y[1] = fma(a5, ry, y[1]); y[2] = fma(a5, rz, y[2]);
        W[0] = fma(a5, xx, W[0]); W[1] = fma(a5, xy, W[1]); W[2] = fma(a5, xz, W[2]);
        W[3] = fma(a5, yy, W[3]); W[4] = fma(a5, yz, W[4]); W[5] = fma(a5, rz * rz, W[5]);
        const double t[7] = {xx * rx, xx * ry, xx * rz, xy * ry, xy * rz, yy * ry, yy * rz};
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            Q[k] = fma(a5, t[k], Q[k]);
            Z[k] = fma(a7, t[k], Z[k]);
        }
    }
};

// H = sum_b f_b Q_ab. as xx xy xz yy yz zz, the entries Q_zz. from the trace tr
__device__ __forceinline__ void adj_contract(const double (&Q)[7], const double (&tr)[3], double fx, double fy, double fz,
                                             double (&H)[6]) {
    const double xzz = tr[0] - Q[0] - Q[3], yzz = tr[1] - Q[1] - Q[5], zzz = tr[2] - Q[2] - Q[6];
    H[0] = Q[0] * fx + Q[1] * fy + Q[2] * fz;
    H[1] = Q[1] * fx + Q[3] * fy + Q[4] * fz;
    H[2] = Q[2] * fx + Q[4] * fy + xzz * fz;
    H[3] = Q[3] * fx + Q[5] * fy + Q[6] * fz;
    H[4] = Q[4] * fx + Q[6] * fy + yzz * fz;
    H[5] = xzz * fx + yzz * fy + zzz * fz;
}

// C[3 a + k] += the pair's matrix for (f, v); s = r.m, m the normal
__device__ __forceinline__ void adj_matrix(double* C, const AdjMoments& M, const double* f, const double* v, double mx,
                                           double my, double mz, double s, double gs, double ts) {
    double H[6];
    {
        const double fx = gs * f[0], fy = gs * f[1], fz = gs * f[2];
        adj_contract(M.Q, M.p, fx, fy, fz, H);
        const double d = fx * M.p[0] + fy * M.p[1] + fz * M.p[2];
        // antisymmetric part p_a f_k - f_a p_k
        const double axy = M.p[0] * fy - fx * M.p[1], axz = M.p[0] * fz - fx * M.p[2], ayz = M.p[1] * fz - fy * M.p[2];
        C[0] += fma(-3.0, H[0], d); C[1] += fma(-3.0, H[1], axy); C[2] += fma(-3.0, H[2], axz);
        C[3] += fma(-3.0, H[1], -axy); C[4] += fma(-3.0, H[3], d); C[5] += fma(-3.0, H[4], ayz);
        C[6] += fma(-3.0, H[2], -axz); C[7] += fma(-3.0, H[4], -ayz); C[8] += fma(-3.0, H[5], d);
    }
    const double c = -6.0 * ts, vx = c * v[0], vy = c * v[1], vz = c * v[2];
    const double s5 = -5.0 * s;
    adj_contract(M.Z, M.y, s5 * vx, s5 * vy, s5 * vz, H);
    const double wx = M.W[0] * vx + M.W[1] * vy + M.W[2] * vz, wy = M.W[1] * vx + M.W[3] * vy + M.W[4] * vz,
                 wz = M.W[2] * vx + M.W[4] * vy + M.W[5] * vz;
    const double d = s * (vx * M.y[0] + vy * M.y[1] + vz * M.y[2]);
    const double yx = s * M.y[0], yy = s * M.y[1], yz = s * M.y[2];
    C[0] += H[0] + d + wx * mx + yx * vx; C[1] += H[1] + wx * my + yx * vy; C[2] += H[2] + wx * mz + yx * vz;
    C[3] += H[1] + wy * mx + yy * vx; C[4] += H[3] + d + wy * my + yy * vy; C[5] += H[4] + wy * mz + yy * vz;
    C[6] += H[2] + wz * mx + yz * vx; C[7] += H[4] + wz * my + yz * vy; C[8] += H[5] + d + wz * mz + yz * vz;
}

__global__ void __launch_bounds__(32 * ADJ_W) adjoint_pairs_kernel(AdjTerm J, int nm, double* partial) {
    constexpr int NC = 9 * ADJ_MAX_MODES;
    __shared__ double sp[ADJ_ST][ADJ_WORDS];  // o (21), c, n, 9 h^2, area, f, v
    __shared__ unsigned char list[ADJ_W][ADJ_TT * ADJ_ST / ADJ_W][2];  // near pairs: lane, source
    __shared__ double sC[ADJ_W][NC][ADJ_TT];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x * ADJ_TT + lane;
    const int s0 = blockIdx.y * ADJ_ST, ns = min(ADJ_ST, J.nS - s0);
    for (int s = threadIdx.x; s < ns; s += 32 * ADJ_W) {
        const PanelRec P = J.src[s0 + s];
        double* d = sp[s];
#pragma unroll
        for (int q = 0; q < 7; ++q)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                d[3 * q + k] = c_rule7[q].l0 * (P.v[k] - P.c[k]) + c_rule7[q].l1 * (P.v[3 + k] - P.c[k]) +
                               c_rule7[q].l2 * (P.v[6 + k] - P.c[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[21 + k] = P.c[k];
            d[24 + k] = P.n[k];
        }
        d[27] = 9.0 * P.h * P.h * (1.0 + 1e-12);
        d[28] = P.area;
        for (int j = 0; j < ADJ_MAX_MODES; ++j)
            for (int a = 0; a < 3; ++a) {
                d[29 + 3 * j + a] = j < nm ? J.f[3 * (long long)(s0 + s) + a + j * J.f_ld] : 0.0;
                d[35 + 3 * j + a] = J.v_src && j < nm ? J.v[3 * (long long)(s0 + s) + a + j * J.v_ld] : 0.0;
            }
    }
    __syncthreads();
    const bool in = t < J.nT;
    const int tt = in ? t : J.nT - 1;
    const double x = J.tgt[3 * tt], y = J.tgt[3 * tt + 1], z = J.tgt[3 * tt + 2];
    double tv[ADJ_MAX_MODES][3];
#pragma unroll
    for (int j = 0; j < ADJ_MAX_MODES; ++j)
#pragma unroll
        for (int a = 0; a < 3; ++a) tv[j][a] = !J.v_src && j < nm ? J.v[3 * (long long)tt + a + j * J.v_ld] : 0.0;
    double C[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) C[k] = 0.0;
    int nnear = 0;
    AdjMoments M;
    for (int s = w; s < ns; s += ADJ_W) {
        const double* d = sp[s];
        const double bx = d[21] - x, by = d[22] - y, bz = d[23] - z;
        bool near = false;
        // within 1e-12 of the threshold and below: the exact test
        if (!(bx * bx + by * by + bz * bz > d[27])) near = rule_of(J.src[s0 + s], x, y, z) != 0;
        near = near && in;
        const unsigned m = __ballot_sync(0xffffffffu, near);
        if (near) {
            unsigned char* e = list[w][nnear + __popc(m & ((1u << lane) - 1))];
            e[0] = (unsigned char)lane;
            e[1] = (unsigned char)s;
        }
        nnear += __popc(m);
        if (near || !in) continue;
        M.zero();
#pragma unroll
        for (int q = 0; q < 7; ++q) M.node(bx + d[3 * q], by + d[3 * q + 1], bz + d[3 * q + 2], c_rule7[q].w);
        const double sm = (bx + d[0]) * d[24] + (by + d[1]) * d[25] + (bz + d[2]) * d[26], gs = J.gs * d[28], ts = J.ts * d[28];
#pragma unroll
        for (int j = 0; j < ADJ_MAX_MODES; ++j)
            if (j < nm)
                adj_matrix(C + 9 * j, M, d + 29 + 3 * j, J.v_src ? d + 35 + 3 * j : tv[j], d[24], d[25], d[26], sm, gs, ts);
    }
    __syncwarp();
    // near pairs by the whole warp: the lanes split the nodes, the sum goes to the target's lane
    for (int n = 0; n < nnear; ++n) {
        const int tl = list[w][n][0], s = list[w][n][1];
        const PanelRec& P = J.src[s0 + s];
        const double* d = sp[s];
        const double X = __shfl_sync(0xffffffffu, x, tl), Y = __shfl_sync(0xffffffffu, y, tl),
                     Zc = __shfl_sync(0xffffffffu, z, tl);
        const double e0x = P.v[0] - X, e0y = P.v[1] - Y, e0z = P.v[2] - Zc;
        const double e1x = P.v[3] - X, e1y = P.v[4] - Y, e1z = P.v[5] - Zc;
        const double e2x = P.v[6] - X, e2y = P.v[7] - Y, e2z = P.v[8] - Zc;
        const int rule = rule_of(P, X, Y, Zc), q1 = rule_off(rule + 1);
        M.zero();
        for (int q = rule_off(rule) + lane; q < q1; q += 32) {
            const QPoint R = d_rule[q];
            M.node(R.l0 * e0x + R.l1 * e1x + R.l2 * e2x, R.l0 * e0y + R.l1 * e1y + R.l2 * e2y,
                   R.l0 * e0z + R.l1 * e1z + R.l2 * e2z, R.w);
        }
        const double sm = e0x * d[24] + e0y * d[25] + e0z * d[26];
        double D[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) D[k] = 0.0;
#pragma unroll
        for (int j = 0; j < ADJ_MAX_MODES; ++j) {
            double vv[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) vv[a] = J.v_src ? d[35 + 3 * j + a] : __shfl_sync(0xffffffffu, tv[j][a], tl);
            if (j < nm) adj_matrix(D + 9 * j, M, d + 29 + 3 * j, vv, d[24], d[25], d[26], sm, J.gs * d[28], J.ts * d[28]);
        }
#pragma unroll
        for (int k = 0; k < NC; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) D[k] += __shfl_xor_sync(0xffffffffu, D[k], o);
            if (lane == tl) C[k] += D[k];
        }
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) sC[w][k][lane] = in ? C[k] : 0.0;
    __syncthreads();
    // the six adjoint vectors: warp w takes outputs w, w + 4, .. of the 6 x modes x 3
    const long long cta = blockIdx.x + (long long)gridDim.x * blockIdx.y;
    for (int e = w; e < ADJ_OUT; e += ADJ_W) {
        const int o = e / (ADJ_MAX_MODES * 3), j = (e / 3) % ADJ_MAX_MODES, k = e % 3;
        const double* lp = J.lam + 3 * (long long)tt + o * J.lam_ld;
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double c = 0.0;
#pragma unroll
            for (int q = 0; q < ADJ_W; ++q) c += sC[q][9 * j + 3 * a + k][lane];
            v = fma(lp[a], c, v);
        }
        if (!in) v = 0.0;
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
        if (lane == 0) partial[cta * ADJ_OUT + e] = v;
    }
}

// out[k] = sum over the ncta partial records in a fixed order: a warp per output
__global__ void __launch_bounds__(1024) adjoint_reduce_kernel(const double* __restrict__ partial, long long ncta,
                                                              double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < ADJ_OUT; k += 32) {
        double s = 0.0;
        for (long long c = lane; c < ncta; c += 32) s += partial[c * ADJ_OUT + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[k] = s;
    }
}

void adjoint_pairs(const AdjTerm* terms, int nterms, int nm, double* out, cudaStream_t st) {
    if (nm < 1 || nm > ADJ_MAX_MODES) fail(SQBEM_ERR_ARG, "adjoint_pairs: %d solutions (at most %d)", nm, ADJ_MAX_MODES);
    init_tables();
    long long total = 0;
    for (int k = 0; k < nterms; ++k)
        total += (long long)ceil_div(terms[k].nT, ADJ_TT) * ceil_div(terms[k].nS, ADJ_ST);
    DevBuf<double> partial((size_t)std::max<long long>(total, 1) * ADJ_OUT, st);
    partial.zero();
    long long off = 0;
    for (int k = 0; k < nterms; ++k) {
        const AdjTerm& J = terms[k];
        if (J.nT <= 0 || J.nS <= 0) continue;
        const dim3 grid(ceil_div(J.nT, ADJ_TT), ceil_div(J.nS, ADJ_ST));
        // far-rule estimate: 83 flops per node for the moments, 160 per solution for its matrix
        const double fl = (double)J.nT * J.nS * (7.0 * 83.0 + 160.0 * nm);
        const double by = (double)J.nS * sizeof(PanelRec) * grid.x + (double)J.nT * 8.0 * 3.0 * 7.0;
        TIMED_LAUNCH("adjoint_pairs", fl, by, adjoint_pairs_kernel, grid, 32 * ADJ_W, 0, st, J, nm,
                     partial.get() + off * ADJ_OUT);
        off += (long long)grid.x * grid.y;
    }
    LAUNCH(adjoint_reduce_kernel, 1, 1024, 0, st, partial.get(), total, out);
}

}  // namespace sqbem
