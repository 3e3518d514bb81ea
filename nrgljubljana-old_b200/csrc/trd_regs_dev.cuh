// Device parts shared by the tridiagonalisation kernels that hold the matrix in
// registers (trd_regs.cu: a cluster per block; trd_grid.cu: many CTAs per block).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "reflector.cuh"

namespace nrgb {
namespace {

namespace trdr {

constexpr int NW = 8;               // warps that hold the matrix
constexpr int NT = 32 * NW;         // their threads

// Sum over the warp: the quads by one FP64 tensor instruction with a matrix
// of ones (two shuffle steps saved), the eight quad sums by shuffles.
__device__ __forceinline__ double warp_sum_mma(double x) {
  double s = 0.0, u = 0.0;
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(s), "+d"(u)
      : "d"(x), "d"(1.0));
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  return s;
}

__host__ __device__ constexpr int pow2_up(int c) { return c <= 1 ? 1 : c <= 2 ? 2 : c <= 4 ? 4 : c <= 8 ? 8 : 16; }

// Shapes of the kernel <KR, C, WR>: rows and columns per CTA it can hold.
template <int KR, int C, int WR>
struct Shape {
  static constexpr int WC = NW / WR;       // column groups of warps
  static constexpr int ROWS = 32 * KR * WR;
  static constexpr int COLS = C * WC;      // columns of a CTA
};

// Sums over the lanes of C columns' partial products: the 32 / pow2_up(C)
// lanes of group g end with column g's sum.
template <int C>
__device__ __forceinline__ double columns_sum(const double (&acc)[C], int lane) {
  constexpr int CP = pow2_up(C);
  double red[CP];
#pragma unroll
  for (int c = 0; c < CP; ++c) red[c] = c < C ? acc[c < C ? c : 0] : 0.0;
  int off = 16;
#pragma unroll
  for (int w2 = CP / 2; w2 >= 1; w2 >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int c = 0; c < w2; ++c) {
      const double keep = up ? red[c + w2] : red[c], send = up ? red[c] : red[c + w2];
      red[c] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    off >>= 1;
  }
#pragma unroll
  for (int o = 16 / CP; o >= 1; o >>= 1) red[0] += __shfl_xor_sync(0xffffffffu, red[0], o);
  return red[0];
}
__device__ __forceinline__ double sum8(const double* p) {
  return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
}

}  // namespace trdr

// Matrix phase of one warp: the rank-2 update of its columns and their
// products with x, over the row chunks KS .. KR-1.  `row`: this lane holds row
// t + 1, in chunk KS, whose updated entries go to Rs.
template <int KS, int KR, int C, int WR>
__device__ __forceinline__ void trdr_update(double (&a)[C][KR], double (&acc)[C], const double (&vj)[C],
                                            const double (&wj)[C], const double2* VW, const double* X, bool row,
                                            double* Rs) {
#pragma unroll
  for (int k = KS; k < KR; ++k) {
    const double2 vw = VW[32 * WR * k];
    const double x = X[32 * WR * k];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      a[c][k] = fma(-vw.y, vj[c], fma(-vw.x, wj[c], a[c][k]));
      acc[c] = fma(a[c][k], x, acc[c]);
    }
  }
  if (row) {
#pragma unroll
    for (int c = 0; c < C; c += 2) *reinterpret_cast<double2*>(Rs + c) = make_double2(a[c][KS], a[c + 1][KS]);
  }
}

// The same from chunk ks on (ks < KR; a warp whose chunks are all done with has nothing to do).
template <int KS, int KR, int C, int WR>
__device__ __forceinline__ void trdr_update_from(int ks, double (&a)[C][KR], double (&acc)[C], const double (&vj)[C],
                                                 const double (&wj)[C], const double2* VW, const double* X, bool row,
                                                 double* Rs) {
  if constexpr (KS < KR) {
    if (ks == KS) trdr_update<KS, KR, C, WR>(a, acc, vj, wj, VW, X, row, Rs);
    else trdr_update_from<KS + 1, KR, C, WR>(ks, a, acc, vj, wj, VW, X, row, Rs);
  }
}

}  // namespace
}  // namespace nrgb
