// Batched FP64 symmetric eigensolver for the invariant-subspace blocks of one
// NRG step (replaces the per-block LAPACK dsyev of src/diag.h:54-89).
//
// Each problem: A (n x n, column-major, both triangles filled) -> eigenvalues
// w (ascending) and orthonormal eigenvectors Z (n x n, column-major, column r
// is the eigenvector of w[r]; ldz == n).  A is destroyed.
//
// Pipeline (all problems of a batch advance together):
//   n <= 32 : the whole solution in one CTA per block (dc_base.cu).
//   n  > 32 : 1) Householder tridiagonalisation with the matrix in registers, up
//                to n = 640 of one thread-block cluster (trd_regs.cu), up to 1776
//                of as many SMs as it needs (trd_grid.cu); the leading columns
//                of larger blocks in panels of 32 (cooperative persistent
//                kernel, trailing rank-64 update on the DMMA GEMM),
//             2) divide and conquer on the tridiagonal (Cuppen splitting,
//                Gu-Eisenstat eigenvectors), subtrees up to 128 rows in one CTA
//                (dc_base.cu), above them merges of equal tree height of all
//                problems in the same launches,
//             3) back-transformation with blocked (WY) reflectors, up to n = 1616 by
//                column slabs in one launch (bt_apply.cu), above on the GEMM.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"

namespace nrgb {

struct SyevDesc {
  int n;
  double* A;   // n x n input (lda = n), destroyed
  double* w;   // n eigenvalues (ascending)
  double* Z;   // n x n eigenvectors (ld = n); must not alias A
};

// Diagonalises a batch of problems whose inputs are ordered on `stream`, and
// returns once the results are complete in device memory.  Implemented by
// the direct solver below and by a server's batcher, which merges the
// batches of several concurrent runs into one solver call.  Returns the
// number of kernel launches made for the batch.  Throws CudaError on failure.
class EigSolver {
 public:
  virtual ~EigSolver() = default;
  virtual int solve(const std::vector<SyevDesc>& probs, cudaStream_t stream) = 0;
  // A run brackets the part of its work that calls solve() (its first
  // sweep); a merging solver waits only for runs inside that part.
  virtual void client_enter() {}
  virtual void client_leave() {}
};

class SyevBatched : public EigSolver {
 public:
  SyevBatched();
  ~SyevBatched();
  int solve(const std::vector<SyevDesc>& probs, cudaStream_t stream) override {
    run(probs, stream);
    return launches_;
  }
  // Solve all problems on `stream`.  Throws CudaError on failure (including
  // a convergence failure or a barrier timeout reported by the kernels).
  void run(const std::vector<SyevDesc>& probs, cudaStream_t stream);
  // Device bytes of workspace that run() will reserve for these sizes.
  static size_t workspace_bytes(const std::vector<int>& n);
  // Launch statistics of the last run().
  int last_launches() const { return launches_; }
  // Largest block the cluster tridiagonalisation holds (0: cluster path off);
  // larger blocks take the many-CTA kernel, and panels before it.
  int cluster_nmax() const { return cl_use(); }
  // The cluster kernel's capacity, before the schedule's limit.
  int cluster_capacity() const { return cl_nmax_; }
  // Bound of the tridiagonalisations' waits: 2^poll_log2 polls of a grid barrier
  // (default 23, about a second) before a wait gives up with an error, at most
  // 2^21 of a word in the many-CTA kernel, 2^12 to 2^20 tries inside a cluster.
  void set_wait_limit(int poll_log2) { wait_log2_ = poll_log2; }
  // Host-side fault injection: while on, every panel launch's barriers
  // expect one CTA more than is launched (a lost CTA) and the other
  // tridiagonalisations a word that nobody sends, so each wait must
  // run out; run() then throws "grid barrier timed out".
  void inject_barrier_shortfall(bool on) { inject_shortfall_ = on; }

 private:
  DeviceArena arena_;
  int* d_err_ = nullptr;
  int* h_err_ = nullptr;  // pinned copy of d_err_
  int launches_ = 0;
  int wait_log2_ = 23;
  bool inject_shortfall_ = false;
  int sms_ = 0;
  int cl_nmax_ = 0;  // largest block it holds (0: cluster path off)
  // blocks up to this size go to the cluster kernel whole: the capacity, or
  // the schedule's limit when it is lower (schedule.cuh)
  int cl_use() const;
  // the many-CTA tridiagonalisation: largest block (0: off) and CTAs of a launch
  int grid_nmax_ = 0, grid_ctas_ = 0;
  // side streams on which the cluster launches of different sizes overlap
  static constexpr int NAUX = 16;
  int naux_ = NAUX;  // side streams in use (NRGB_SIDE_STREAMS, for comparisons)
  cudaStream_t aux_[NAUX] = {};
  cudaEvent_t fork_ = nullptr, join_[NAUX] = {};
  // blocks up to 32 run beside the larger blocks' work
  cudaStream_t small_st_ = nullptr;
  cudaEvent_t small_done_ = nullptr;
};

}  // namespace nrgb
