// Back-transformation of eigenvectors by the reflectors of the
// tridiagonalisation, one column slab per CTA (bt_apply.cu).
#pragma once
#include <cuda_runtime.h>

namespace nrgb {

constexpr int BT_NB = 64;  // reflectors of a compact WY block

struct BtSlabProb {
  const double* A;    // n x n (ld n): reflector c below the subdiagonal of column c (v[c + 1] = 1)
  const double* tau;  // n-1
  double* T;          // ceil((n-1)/64) blocks of 64 x 64: the WY factors
  double* Z;          // n x n (ld n): eigenvectors of T in, of A out
  int n;
  int blk0, cta0;     // first block of the WY launch, first CTA of the slab launch
};

// Largest block the slab kernel takes.
int bt_slab_nmax();
// Columns of a slab, from the total number of columns of the launch's blocks
// and the largest block.
int bt_slab_columns(long columns, int nmax);

// WY factors of every block of 64 reflectors (`blocks` CTAs in all).
cudaError_t bt_wy_launch(const BtSlabProb* d, int nprob, int blocks, cudaStream_t st);
// Z <- H_0 H_1 ... H_{n-2} Z, `ctas` slabs of `columns` columns in all.
cudaError_t bt_apply_launch(const BtSlabProb* d, int nprob, int columns, int ctas, int nmax, cudaStream_t st);

}  // namespace nrgb
