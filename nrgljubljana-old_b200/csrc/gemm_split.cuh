// Split-precision grouped GEMM: FP64 products computed as exact INT8
// tensor-core products (tcgen05.mma kind::i8, INT32 accumulators in tensor
// memory) with FP64 recombination.
//
//   C_p = beta_p * C_p + sum_{s in segments(p)} alpha_s * op(A_s) op(B_s)
//
// Same problem/segment description as the FP64 grouped GEMM (GemmProb,
// GemmSeg; column-major, op = as stored or transposed).  `slices` asks for the
// precision of that many truncated 7-bit slices per operand.  Each row i of
// op(A) is scaled by a power of two 2^eA_i (and each column j of op(B) by
// 2^eB_j) so that its entries lie in (-1, 1), rounded to 8 D - 1 bits and cut
// into D = slices balanced 8-bit digits:
//   op(A)_il = 2^eA_i sum_{p=1..D} a^(p)_il 2^(1-8p) + r_il,
// |r_il| <= 2^(eA_i - 8D)  (Ozaki-type splitting, Ozaki, Ogita, Oishi and
// Rump 2012, with integer slices as in the INT8 emulation of DGEMM).  The
// balanced digits reach 0.996 of the power of two; a row whose largest entry is
// nearer to it is scaled by the next one.  Every digit product a^(p) b^(q) is
// exact in INT32; the products with the same p + q share one accumulator;
// products with p + q > D + 1 are dropped (they lie at the rounding's level).
// The D accumulators are recombined exactly in 64-bit integers, rounded once to
// FP64 and scaled by 2^(eA_i + eB_j).  The error per entry is bounded by about
// k * 2^(eA_i + eB_j) * 2^(-8D) * (D + 2) and the rounding of the result; a
// scale is at most 2.01 times its row's largest entry.
// Seven digits for 8 slices (28 products instead of 36) hold what eight truncated
// slices do in most rows, but a bit less in those scaled by the next power of two:
// products of such rows and columns were twice as far off as with the slices
// (0.999 in each, K = 400: 21.8 against 11.9 units of 2^-53 of the largest
// entries' product).
//
// This replaces the BLAS gemm calls of the operator recalculation
// (src/recalc.cc:90-91, 268-272) and of the density matrices
// (src/dmnrg.h:382-387) in the split-precision form of a run.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"
#include "gemm_f64.cuh"

namespace nrgb {

constexpr int SPLIT_MIN_SLICES = 2;
constexpr int SPLIT_MAX_SLICES = 8;
// Largest inner dimension of one segment: the accumulator of p + q = d sums
// d - 1 <= 8 digit products of magnitude <= 128^2 k, which must stay below
// 2^31.  Longer segments are cut into pieces of this length.
constexpr int SPLIT_MAX_K = 16000;

// Device bytes of workspace that split_gemm_grouped needs for these
// problems (host descriptors, as for the FP64 launch).
size_t split_gemm_workspace(const GemmProb* probs, int nprob, const GemmSeg* segs, int slices);

// Slice every segment's operands into `ws` (reset by the caller; it must
// hold split_gemm_workspace bytes) and launch the tensor-core products.
// `tag` names the call site in the launch accounting.  Throws CudaError.
void split_gemm_grouped(const GemmProb* probs, int nprob, const GemmSeg* segs, int slices, DeviceArena& ws,
                        cudaStream_t st, const char* tag = "gemm_i8");

// Error flag of the split kernels' bounded waits (nonzero: a wait gave up);
// read and cleared by the host after a synchronisation.
int split_gemm_take_error(cudaStream_t st);

}  // namespace nrgb
