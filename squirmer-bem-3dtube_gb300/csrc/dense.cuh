// dense.cuh -- dense linear algebra on the GPU for the BEM systems.
//
// Replaces the LAPACK/BLAS calls of the reference (src/utils/linalg.hpp:17-78):
//   gemm      -> dgemm_          C = alpha op(A) op(B) + beta C, column-major
//   LUFactor  -> dgetrf_/dgetrs_ LU with partial pivoting and solves
//   solve     -> dgesv_          (factor + solve)
//
// LU design.  Partial pivoting on the BEM blocks of this problem never swaps a
// row (the matrices are diagonally dominant in the pivoting sense), so the
// factorisation runs a blocked right-looking LU WITHOUT row exchanges and
// certifies on the fly that partial pivoting would have chosen the same pivots:
// dgetrf keeps the diagonal pivot exactly when no multiplier exceeds 1 in
// magnitude (idamax returns the first maximum, so ties keep the diagonal).  If
// any |l_ij| > 1 (or a pivot is zero) the certificate fails and the matrix is
// refactored from a saved copy by an unblocked partial-pivoting LU that swaps
// rows exactly like dgetrf.  Either way the factors and pivots are those of
// dgetrf up to rounding.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"

namespace sqbem {

constexpr int LU_NB = 256;  // panel width of the blocked LU (FP64)

// The word that a bounded wait of the tensor-core products sets when it runs out, for the
// calls of one stream.
struct WaitError {
    DevBuf<int> w;
    int* get(cudaStream_t st);  // the word, zeroed at first use
    void check();               // waits for the stream; SQBEM_ERR_TIMEOUT if a wait ran out
};

// C(MxN) = alpha * op(A) * op(B) + beta * C   (column-major, FP64).  With err (a
// WaitError's word, checked by the caller) large products run as digit products on the
// tensor cores (oz_gemm.cuh); C must not overlap A or B.
void gemm64(bool ta, bool tb, int M, int N, int K, double alpha, const double* A, long long lda,
            const double* B, long long ldb, double beta, double* C, long long ldc, cudaStream_t st,
            int* err = nullptr);

// The same for at most SK_N columns and tb = false, for a batch of matrices at the strides
// sa, sb, sc.
constexpr int SK_N = 8;
void gemm64_few(bool ta, int M, int N, int K, double alpha, const double* A, long long lda, const double* B,
                long long ldb, double beta, double* C, long long ldc, cudaStream_t st, int batch = 1,
                long long sa = 0, long long sb = 0, long long sc = 0);

// y = recip(x) elementwise on device arrays: the reciprocal of the LU kernels (tested through
// sqbem_test_recip)
void recip_eval(int n, const double* x, double* y, cudaStream_t st);

// C (m x 6) = A K, K the rigid-body map of np panels with the offsets r (3 per panel) from the
// centre; A is m x 3 np.
void rigid64(int m, int np, const double* A, long long lda, const double* r, double* C, long long ldc, cudaStream_t st);

// LU factorisation (dgetrf semantics) of an n x n column-major matrix, kept on
// the device with the inverses of its diagonal blocks (used by the solves).
struct LU64 {
    int n = 0;
    long long ld = 0;
    DevBuf<double> A;      // factors (unit L below the diagonal, U on and above)
    DevBuf<double> Linv;   // per diagonal block: inverse of the unit-lower block (LU_NB x LU_NB)
    DevBuf<double> Uinv;   // per diagonal block: inverse of the upper block
    DevBuf<int> ipiv;      // 0-based pivot rows (dgetrf convention, only if pivoted)
    bool pivoted = false;  // true if the certificate failed and rows were exchanged

    // Factor M (n x n, leading dimension ld, device); M is copied.
    // Throws Error(SQBEM_ERR_SINGULAR, what) on a zero pivot.
    void factor(const double* M, int n, long long ld, cudaStream_t st, const char* what);
    // Take ownership of a device buffer (n x n, leading dimension n) and factor it in place.
    void factor_inplace(DevBuf<double>&& M, int n, cudaStream_t st, const char* what);
    // B <- A^{-1} B for B (n x nrhs, leading dimension ldb, device); err as in gemm64
    void solve(double* B, long long ldb, int nrhs, cudaStream_t st, int* err = nullptr) const;
    // B <- (leading m x m block of A)^{-1} B from the same factor; not after exchanges
    void solve_leading(int m, double* B, long long ldb, int nrhs, cudaStream_t st) const;
    // B <- A^{-T} B (dgetrs 'T'): U^T then L^T solves, then the row exchanges undone
    void solve_transpose(double* B, long long ldb, int nrhs, cudaStream_t st) const;
};

// Solve with the certified LU; helpers shared with the mixed path.
void copy_matrix64(const double* src, long long lds, double* dst, long long ldd, int rows, int cols, cudaStream_t st);
// max |A| over a column-major block (result written to *out on the device)
void max_abs64(const double* A, long long lda, int rows, int cols, double* out, cudaStream_t st);

}  // namespace sqbem
