// oz_gemm.cuh -- FP64 matrix products on the BF16 tensor cores (tcgen05).
//
// Every row of A and every column of B is scaled by its own power of two to
// 64-bit fixed point and cut into eight signed base-256 digits, d_0 (most
// significant) .. d_7, |d_i| <= 128: small integers, exact in BF16 (the error-free
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication", Numer. Algorithms 59, 2012).  A product of two digits is
// at most 2^14, so sums of them are exact in the FP32 accumulators up to 2^24.
// The 36 digit products with i + j <= 7 are summed by their weight i + j, each sum
// is read back as an integer, all of them are added in two 64-bit integers and the
// 96-bit total is rounded to FP64 once.  What is dropped lies below 2^-60 of the
// row's largest entry times the column's, against the FP64 loop's rounding of
// every partial sum.
//
// The FP64 loop does not see powers of two that move from A's column k to B's row k; a fixed
// point does.  An LU of a matrix whose rows have different scales has small multipliers that
// meet large entries, and kept 2^-62 of the largest multiplier: rows 2^-40 apart gave
// solutions good to 1e-7.  So oz_product first scales every k by a power of two after which
// the rows of B (its columns taken relative to their largest entries) have equal largest
// exponents; the scales change the fixed points only, and cancel in the products.  It
// takes one more pass over B; a product whose operands are known to be even (the Fourier blocks)
// does without (split and oz_gemm).
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace sqbem {

// Digits of an operand: rows x k values (the rows of A, or the columns of B) as
// blocks of 128 rows x 16 k x 8 digits (32 KB), each digit's 128 x 16 BF16 in the
// tensor cores' no-swizzle order (two halves of 8 k, 16 bytes per row), zero
// padded; the biased exponent of every row's largest entry beside them.
struct OzMat {
    DevBuf<uint4> d;
    DevBuf<int> ex;
    int rows = 0, k = 0, k16 = 0, batch = 1, block = 128;
    bool right = false;
    // the values' source, for rows that hold an infinity or a NaN
    const double* src = nullptr;
    long long rs = 0, ks = 0, bs = 0;
    // element (r, c) of matrix b is a[r * rs + c * ks + b * bs]; `right` where the operand is B
    // (blocks of 64 rows then, while k <= 256); q: scales along k (oz_scales), the same for A and B
    void split(const double* a, long long rs, long long ks, int rows, int k, cudaStream_t st, bool right = false,
               int batch = 1, long long bs = 0, const int* q = nullptr);
    // its two halves: sizes and buffers, then the digits
    void lay_out(const double* a, long long rs, long long ks, int rows, int k, cudaStream_t st, bool right,
                 int batch = 1, long long bs = 0);
    void split_values(const int* q, cudaStream_t st);
};

// C (M x N, column-major) = alpha A B + beta C for the digits of A (M rows) and of
// B (N columns, given as rows) over the same k, for every matrix of the batch (C at
// stride cb).  The sources of A and B must be alive and unchanged until the launch has
// run; C may be one of them, but must not overlap them otherwise.  A row or a column with an
// infinity or a NaN gives the plain sums of its elements, or NaN where C is a source, and leaves the
// others as they are.  *err is set if a bounded wait expires
// (SQBEM_ERR_TIMEOUT to the caller).
void oz_gemm(const OzMat& A, const OzMat& B, double alpha, double beta, double* C, long long ldc, int* err,
             cudaStream_t st, long long cb = 0);

// The scales along k of a product with B (element (k, n) at B[n * rs + k * ks]) into the K words
// of q, which are zero before.
void oz_scales(const double* B, long long rs, long long ks, int N, int K, int* q, cudaStream_t st);

// C = alpha A B + beta C from the values, with scales along k: element (m, k) of A at A[m * ars + k * aks],
// (k, n) of B at B[n * brs + k * bks]; C as in oz_gemm.  q (may be null): K words of zeros for the scales.
void oz_product(const double* A, long long ars, long long aks, const double* B, long long brs, long long bks, int M, int N,
                int K, double alpha, double beta, double* C, long long ldc, int* err, cudaStream_t st, int* q = nullptr);

}  // namespace sqbem
