// The PCA's dense FP64 steps on blocks of up to 64 columns (kg_dense.cu): a Krylov block's
// orthonormalisation as one cluster kernel, and Householder QR + Jacobi for the blocks it
// cannot take.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace kg {

constexpr uint32_t kQrMaxCols = 64;

// The thin SVD of `rest` (g x w column-major f64, w <= 64, g >= w; left as it is): u (g x w)
// the left singular vectors, out[0 .. w) the singular values (descending, ties to the lower
// column), out[w] = |block|_F of the g x w `block`, out[w + 1] = 0, or 1 if a Cholesky pivot
// was not positive (a numerically rank-deficient block: use qr_svd) or Jacobi did not
// converge. q: g x w scratch.
void extend_svd(const double* block, const double* rest, uint32_t g, uint32_t w, double* q,
                double* u, double* out, cudaStream_t s);

// The same SVD by Householder QR and Jacobi on R in one CTA (`b` is overwritten): u,
// out[0 .. w) and out[w + 1] as above; out[w] is left as it is.
void qr_svd(double* b, uint32_t g, uint32_t w, double* u, double* out, cudaStream_t s);

}  // namespace kg
