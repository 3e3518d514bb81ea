// Unblocked Householder tridiagonalisation of one block per thread-block
// cluster, the matrix held in the CTAs' registers (trd_regs.cu).
#pragma once
#include <cuda_runtime.h>

namespace nrgb {

struct TrdClProb {
  double* A;    // n x n, leading dimension ld: input; on return the reflectors below the subdiagonal
  double* d;    // n
  double* e;    // n-1
  double* tau;  // n-1
  int n;
  int ld;
};

// The kernel a block of size n takes: a shape (rows and columns per CTA) and
// the CTAs of its cluster.  shape < 0: no shape holds it.
struct TrdrGroup {
  int shape, cl;
};
TrdrGroup trdr_group(int n);

// Prepares the current device (function attributes; the values are the same
// for every caller) and returns the largest block the shapes hold there
// (0: clusters not usable).
int trdr_init();

// Tridiagonalises `nprob` blocks of one group.  *fail is set when a wait
// inside a cluster gave up, after 2^wait_log2 tries of about a microsecond.
// expect_extra: the waits expect so many words that no CTA sends (0; 1 injects
// a lost message).
cudaError_t trdr_launch(TrdrGroup g, const TrdClProb* d, int nprob, int wait_log2, int expect_extra, int* fail,
                        cudaStream_t st);

}  // namespace nrgb
