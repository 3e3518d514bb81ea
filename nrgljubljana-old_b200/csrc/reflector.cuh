// The Householder reflector of a column, in the range where its squares underflow.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace nrgb {
namespace {

// beta, tau and the scale of v (v = x scale) of the reflector of a column with the
// entry alpha below the diagonal and the squared norm nn of x, the rest.
__device__ __forceinline__ void reflector(double alpha, double nn, double& beta, double& tau, double& scale) {
  beta = alpha;
  tau = scale = 0.0;
  if (nn != 0.0) {
    beta = -copysign(sqrt(fma(alpha, alpha, nn)), alpha);
    tau = (beta - alpha) / beta;
    scale = 1.0 / (alpha - beta);
  }
}

// The squares of a column's entries have lost digits to underflow: its reflector
// would not be orthogonal.  What a matrix of low rank leaves behind its first
// columns is rounding of rounding, 1e-16 of the column before, so that such
// columns occur in matrices of any size and scale (all ones, n = 21: eigenvectors
// orthogonal to 4e-3).  Their norm is formed again from scaled entries.  (nn is not
// zero, so some |x| is at least 1e-162; a norm whose square underflows to zero is
// zero as far as the matrix's other columns are concerned.)
__device__ __forceinline__ bool squares_lost(double alpha, double nn) {
  return nn != 0.0 && fma(alpha, alpha, nn) < 0x1p-960;
}
// Power of two that brings the larger of |alpha| and the largest |x| to [1, 2)
// (at most 2^1022), from their upper words.
__device__ __forceinline__ int upper_word(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ double small_scale(double alpha, int xtop, double& inverse) {
  const int e = max(max(upper_word(alpha), xtop) >> 20, 1);
  inverse = __hiloint2double(e << 20, 0);
  return __hiloint2double((2046 - e) << 20, 0);
}
// The same with nn from x p, p = 1 / inverse (small_scale).
__device__ __forceinline__ void reflector_small(double alpha, double nn, double p, double inverse, double& beta,
                                                double& tau, double& scale) {
  reflector(alpha * p, nn, beta, tau, scale);
  beta *= inverse;
  scale *= p;
}

}  // namespace
}  // namespace nrgb
