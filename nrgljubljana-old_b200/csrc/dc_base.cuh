// Divide and conquer of small tridiagonal problems inside one CTA (dc_base.cu).
#pragma once
#include <cuda_runtime.h>

namespace nrgb {

constexpr int DC_BASE = 128;  // largest subtree one CTA solves

// Rows [lo, lo + s) of a tridiagonal matrix of size n, torn from its neighbours
// (Cuppen); s <= DC_BASE.
struct DcBaseProb {
  const double* d;  // n
  const double* e;  // n-1
  double* D;        // n: eigenvalues of the subtree, ascending, at [lo, lo + s)
  double* Q;        // n x n (ld n): its eigenvectors at [lo, lo + s) x [lo, lo + s)
  int n, lo, s;
};
// smax: the largest s.  *fail is set to 1 when a secular equation did not converge.
cudaError_t dc_base_launch(const DcBaseProb* d, int nprob, int smax, int* fail, cudaStream_t st);

// Whole eigen-decompositions of symmetric blocks up to 32 x 32, a CTA each.
constexpr int SYEV_TINY = 32;
struct TinyProb {
  const double* A;  // n x n
  double* w;        // n, ascending
  double* Z;        // n x n
  int n;
};
// Up to TINY_INLINE descriptors are taken from the host (d null), more from the
// device.
constexpr int TINY_INLINE = 96;
cudaError_t syev_tiny_launch(const TinyProb* h, const TinyProb* d, int nprob, int* fail, cudaStream_t st);

}  // namespace nrgb
