// circulant64.cuh -- FP64 solves with a matrix that is n_theta-fold rotationally symmetric.
//
// The tube's deflated single-layer block (and the duct's system) couple panels that a
// rotation by one sector maps onto each other (tube_sym.cuh).  With every panel's
// 3-vectors in the frame of its sector the matrix is block-circulant, and a Fourier
// transform over the sectors leaves n_theta / 2 + 1 complex blocks of order 3 nb
// (tube_fourier.cuh).  Here the blocks, their inverses and the transforms are FP64: an FP32
// Gauss-Jordan inverse X of each block C is the start of the Newton-Schulz iteration
//     X <- X + X (I - C X)
// (G. Schulz, ZAMM 13, 1933), whose error squares at every step, with the products on
// the tensor cores (oz_gemm.cuh).  Y = T^{-1} X then takes two transforms and one product per
// frequency, of order 6 nb, where the LU of T takes 2 (3 Nt)^2 operations per column.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"
#include "oz_gemm.cuh"
#include "tube_sym.cuh"

namespace sqbem {

struct Circulant64 {
    int nth = 0, nb = 0, nf = 0;  // sectors, panels per sector, frequencies held
    int n3 = 0, m2 = 0, nt = 0;   // block order 3 nb, its real form's 2 n3, 3 Nt
    DevBuf<int> panel;            // nb x nth, as in TubeSymmetry
    DevBuf<double> inv;           // nf inverses in real form [[Re, -Im], [Im, Re]], m2 x m2 column-major
    OzMat digits;                 // of the inverses, for many columns
    bool ready = false;

    // From the rows of sector 0 (3 nb x 3 Nt, column-major, leading dimension 3 nb).  False,
    // and not ready, if a block has a zero pivot or the iteration has not converged.  Waits
    // for the stream; *tie (may be null) is a device flag downloaded with the rest.
    bool build(const TubeSymmetry& sym, const double* T0, const int* tie, cudaStream_t st);
    // B <- T^{-1} B, or T^{-T} B, for B (3 Nt x nrhs); err as in gemm64
    void solve(double* B, long long ldb, int nrhs, cudaStream_t st, int* err, bool transpose = false) const;
};

// Whether FP64 solves take this path: symmetry found, n_theta and block order within the
// kernels' limits, not switched off (SQBEM_TUBE_SYMMETRY=0, SQBEM_TUBE_FOURIER=0).
bool circulant64_supported(const TubeSymmetry& sym);

// The rows of sector 0 of a rotationally symmetric panel set: SL / (8 pi mu) into S and, if D
// is not null, -DL / (8 pi) into D (each 3 nb x 3 P, column-major, leading dimension 3 nb).
// *tie is set if a pair lies so close to a quadrature threshold that its rotated copies
// might take another rule (relative 1e-11): the caller then assembles every pair.
void assemble_sector0(const std::vector<PanelRec>& host, const PanelRec* dev, const TubeSymmetry& sym, double mu,
                      double* S, double* D, int* tie, cudaStream_t st);

// S[3a + al, 3q + b] += sc n_rep(a)[al] n_q[b] area_q: the deflation of those rows
void deflate_sector0(double* S, const PanelRec* dev, const TubeSymmetry& sym, int P, double sc, cudaStream_t st);

// Frequency 0: M (3 nb x 3 nb, column-major) = sum_d T0[:, panel(:, d)] R_d, what T does to
// vectors that every rotation maps onto themselves
void fold_sector0(const double* T0, const int* panel, int nth, int nb, double* M, cudaStream_t st);

}  // namespace sqbem
