// The PCA's dense FP64 steps on blocks of up to 64 columns (kg_dense.cu).
#pragma once

#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

namespace kg {

constexpr uint32_t kQrMaxCols = 64;

// One step of shifted CholeskyQR3 (Fukaya, Kannan, Nakatsukasa, Yamamoto and Yanagisawa,
// "Shifted Cholesky QR for computing the QR factorization of ill-conditioned matrices",
// SIAM J. Sci. Comput. 2020), w <= 64: the upper Cholesky factor R of the Gram matrix G
// (w x w, column-major) plus shift * trace(G) on the diagonal (trace(G) = |A|_F^2 >=
// |A|_2^2), into r (w x w column-major, zeros below). *status = 1 (and r left as it is) if
// a pivot is not positive (the caller then uses Householder QR).
void cholesky_step(const double* gram, uint32_t w, double shift, double* r, int* status,
                   cudaStream_t s);

// The parts that a block's n values' sum of squares comes in.
inline uint32_t squares_parts(uint64_t n) {
  return (uint32_t)std::min<uint64_t>(128, n / 16384 + 1);
}

// The SVD of R = R_3 R_2 R_1, the steps' factors one after another in r (w x w upper
// triangular, column-major, w <= 64): out[0 .. w) the singular values (descending, ties to
// the lower column), u_r (w x w: column c the unit left singular vector of out[c]; zero for
// 0), out[w] = 0, or 1 if Jacobi did not converge or *status is set: then a step's factor is not
// there, r is not read, and the singular values and u_r are left as they are. And from out[w + 1]
// on: the squares_parts(n) parts of the sum of squares of `block` (n values).
void small_svd(const double* r, uint32_t w, const double* block, uint64_t n, const int* status,
               double* u_r, double* out, cudaStream_t s);

// The thin SVD of the g x w column-major block `b` (overwritten): u the left singular
// vectors, out[0 .. w] as above.
void qr_svd(double* b, uint32_t g, uint32_t w, double* u, double* out, cudaStream_t s);

// The squares_parts(n) parts of the sum of squares of m (n values).
void squares(const double* m, uint64_t n, double* out, cudaStream_t s);

// The `take` largest eigenvalues of the symmetric m x m matrix `a` (column-major, both halves),
// descending, into `values`, and their orthonormal vectors into `vectors` (m x take,
// column-major) (kg_eigen.cu). False, with both undefined and `a` as it was, where it does not
// apply (m past 544, take past 50, no room for a cluster of 16 CTAs) or where the pairs fail their
// check (residuals of the norm and orthonormality within (16 + m / 8) 2^-52). Waits for the stream.
bool leading_eigenpairs(cublasHandle_t cublas, const double* a, uint32_t m, uint32_t take,
                        double* vectors, std::vector<double>& values, cudaStream_t s);

}  // namespace kg
