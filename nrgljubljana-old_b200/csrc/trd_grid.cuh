// Unblocked Householder tridiagonalisation of blocks beyond one cluster, the
// matrix held in the registers of up to every SM (trd_grid.cu).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace nrgb {

struct TrdGridProb {
  double* A;    // n x n, leading dimension ld: input; on return the reflectors below the subdiagonal
  double* d;    // n
  double* e;    // n-1
  double* tau;  // n-1
  double* ex;   // exchange buffer, trd_grid_exchange(n) doubles, zero on entry
  int n;
  int ld;
  int wait_log2;     // a wait gives up after 2^wait_log2 polls
  int expect_extra;  // 1 injects an entry that no CTA ever writes
  int shape, cta0, ncta;  // set by trd_grid_place
};

// Doubles of one of the two exchange buffers of a block of size n (two entries
// a column, one never written, one a CTA), and of both.
constexpr int TRD_GRID_CTAS = 256;  // most CTAs of a block
__host__ __device__ constexpr size_t trd_grid_stride(int n) { return 4 * ((size_t)n + 1) + 2 * TRD_GRID_CTAS; }
inline size_t trd_grid_exchange(int n) { return 2 * trd_grid_stride(n); }

// Prepares the current device and returns the largest block the kernel holds
// there (0: no cooperative launches); *ctas: the CTAs one launch may have.
int trd_grid_init(int* ctas);

// CTAs a block of size n takes.
int trd_grid_ctas(int n);

// Sets shape, cta0 and ncta of the blocks of one launch; their CTAs' sum.
int trd_grid_place(std::vector<TrdGridProb>& probs);

// One cooperative launch of `nprob` placed blocks on `ctas` CTAs.  *fail is
// set when a wait gave up.
cudaError_t trd_grid_launch(const TrdGridProb* d, int nprob, int ctas, int* fail, cudaStream_t st);

}  // namespace nrgb
