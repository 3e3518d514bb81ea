// Back-transformation of the eigenvectors, Z <- H_0 H_1 ... H_{n-2} Z, for
// blocks whose column slab fits a CTA's shared memory.
//
// The columns of Z are independent, so a CTA keeps a slab of them in shared
// memory and applies every block of 64 reflectors to it, last block first,
// Z[r0:, :] -= V (T (V^T Z[r0:, :])), without meeting another CTA: one launch in
// place of three grouped GEMMs per 64 reflectors, whose few tiles left most
// SMs idle and whose K loops were a chain of 64 x 64 x 16 steps.  What bounds it
// is the FP64 tensor pipe of the SMs that have a slab, and for larger blocks the
// reading of V (4 n^2 bytes a slab) from L2.
// All three products run on the FP64 tensor instruction m8n8k4; V and T come
// straight from L2 in fragment layout (V^T fragments are 8 columns x 32 bytes, V
// fragments 4 columns x 64 bytes: whole sectors), the next 8 fragments loaded
// while the current ones multiply.
#include <math.h>

#include <algorithm>

#include "bt_apply.cuh"
#include "common.cuh"

namespace nrgb {

namespace {

constexpr int NT = 256, NWARP = NT / 32;
constexpr int XLD = BT_NB + 4;  // row stride of X, Y in shared memory ([column][reflector])

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Entry (row, c) of V: reflector c, 1 in row c + 1, zero above.
__device__ __forceinline__ double ldv(const double* __restrict__ A, int n, int row, int c) {
  if (row > c + 1 && row < n) return __ldg(A + row + (size_t)c * n);
  return (row == c + 1 && row < n) ? 1.0 : 0.0;
}

__host__ __device__ inline int slab_ld(int n) { return ((n + 15) & ~15) + 4; }
__host__ __device__ inline size_t slab_smem(int n, int columns) {
  return ((size_t)columns * slab_ld(n) + 2 * (size_t)columns * XLD) * sizeof(double);
}

__device__ __forceinline__ int find_prob(const BtSlabProb* probs, int nprob, int b, bool wy) {
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((wy ? probs[mid].blk0 : probs[mid].cta0) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One CTA per block of 64 reflectors: G = V^T V (its upper tiles) on the tensor
// pipe, then the recurrence T[0:j, j] = -tau_j T[0:j, 0:j] G[0:j, j] (dlarft)
// with four threads per row.  Runs beside the divide and conquer, which does
// not need it.
__global__ void __launch_bounds__(NT) bt_wy_kernel(const BtSlabProb* __restrict__ probs, int nprob) {
  extern __shared__ double sm[];
  double(*Ts)[BT_NB + 1] = reinterpret_cast<double(*)[BT_NB + 1]>(sm);
  double(*Gs)[BT_NB + 1] = reinterpret_cast<double(*)[BT_NB + 1]>(sm + BT_NB * (BT_NB + 1));
  const BtSlabProb P = probs[find_prob(probs, nprob, blockIdx.x, true)];
  const int k = blockIdx.x - P.blk0, n = P.n, j0 = k * BT_NB, nb = min(BT_NB, n - 1 - j0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  double acc[8][2];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q][0] = acc[q][1] = 0.0;
  for (int r = j0 + 1; r < n; r += 4) {
    double f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = j0 + 8 * q + g;
      f[q] = c < n - 1 ? ldv(P.A, n, r + t, c) : 0.0;
    }
    double a = f[0];
#pragma unroll
    for (int q = 1; q < 8; ++q) a = warp == q ? f[q] : a;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q >= warp) dmma(acc[q][0], acc[q][1], a, f[q]);
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      Gs[8 * warp + g][8 * q + 2 * t + h] = acc[q][h];
      Ts[8 * warp + g][8 * q + 2 * t + h] = 0.0;
    }
  __syncthreads();
  const int i = tid >> 2, q = tid & 3;
  for (int j = 0; j < nb; ++j) {
    double s = 0.0;
    for (int l = i + q; l < j; l += 4) s += Ts[i][l] * Gs[l][j];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    // column j is written here and read only from step j+1 on
    if (q == 0) {
      const double tj = P.tau[j0 + j];
      if (i < j) Ts[i][j] = -tj * s;
      else if (i == j) Ts[j][j] = tj;
    }
    __syncthreads();
  }
  double* T = P.T + (size_t)k * BT_NB * BT_NB;
  for (int idx = tid; idx < BT_NB * BT_NB; idx += NT) T[idx] = Ts[idx % BT_NB][idx / BT_NB];
}

// One CTA per slab of 8 CT columns of Z.
template <int CT>
__global__ void __launch_bounds__(NT) bt_apply_kernel(const BtSlabProb* __restrict__ probs, int nprob) {
  constexpr int NC = 8 * CT;
  extern __shared__ double sm[];
  const BtSlabProb P = probs[find_prob(probs, nprob, blockIdx.x, false)];
  const int n = P.n, c0 = (blockIdx.x - P.cta0) * NC, ldz = slab_ld(n);
  double* Zs = sm;                   // [NC][ldz]
  double* Xs = Zs + NC * ldz;        // [NC][XLD]
  double* Ys = Xs + NC * XLD;        // [NC][XLD]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (int c = 0; c < NC; ++c)
    for (int i = tid; i < ldz; i += NT) Zs[c * ldz + i] = (i < n && c0 + c < n) ? P.Z[i + (size_t)(c0 + c) * n] : 0.0;
  __syncthreads();
  for (int k = (n - 2) / BT_NB; k >= 0; --k) {
    const int j0 = k * BT_NB, r0 = j0 + 1;
    // X = V^T Z: warp w forms the rows (reflectors) 8 w .. 8 w + 7
    {
      double acc[2][CT][2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < CT; ++q) acc[h][q][0] = acc[h][q][1] = 0.0;
      const int c = j0 + 8 * warp + g;
      const bool on = c < n - 1;
      const int rb = (r0 + 8 * warp) & ~3;  // rows above are zero in these reflectors
      double f[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) f[u] = on ? ldv(P.A, n, rb + 4 * u + t, c) : 0.0;
      for (int r = rb; r < n; r += 32) {
        double fn[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) fn[u] = on ? ldv(P.A, n, r + 32 + 4 * u + t, c) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int row = min(r + 4 * u + t, ldz - 1);
#pragma unroll
          for (int q = 0; q < CT; ++q)
            dmma(acc[u & 1][q][0], acc[u & 1][q][1], f[u], Zs[(8 * q + g) * ldz + row]);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) f[u] = fn[u];
      }
#pragma unroll
      for (int q = 0; q < CT; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) Xs[(8 * q + 2 * t + h) * XLD + 8 * warp + g] = acc[0][q][h] + acc[1][q][h];
    }
    // T's fragments (upper triangular) arrive while the others finish
    double ft[BT_NB / 4];
    const double* T = P.T + (size_t)k * BT_NB * BT_NB;
#pragma unroll
    for (int u = 0; u < BT_NB / 4; ++u)
      ft[u] = 4 * u + 3 >= 8 * warp ? __ldg(T + (8 * warp + g) + (size_t)(4 * u + t) * BT_NB) : 0.0;
    __syncthreads();
    // Y = T X
    {
      double acc[CT][2];
#pragma unroll
      for (int q = 0; q < CT; ++q) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
      for (int u = 0; u < BT_NB / 4; ++u)
        if (4 * u + 3 >= 8 * warp) {
#pragma unroll
          for (int q = 0; q < CT; ++q) dmma(acc[q][0], acc[q][1], ft[u], Xs[(8 * q + g) * XLD + 4 * u + t]);
        }
#pragma unroll
      for (int q = 0; q < CT; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) Ys[(8 * q + 2 * t + h) * XLD + 8 * warp + g] = -acc[q][h];
    }
    __syncthreads();
    // Z[r0:, :] += V (-Y): row tiles of 8 over the warps
    {
      const int m0 = r0 & ~7;
      double f[16];
      int m = m0 + 8 * warp;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int c = j0 + 4 * u + t;
        f[u] = c < n - 1 ? ldv(P.A, n, m + g, c) : 0.0;
      }
      for (; m < n; m += 8 * NWARP) {
        double acc[CT][2], fn[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int c = j0 + 4 * u + t;
          fn[u] = c < n - 1 ? ldv(P.A, n, m + 8 * NWARP + g, c) : 0.0;
        }
        const int row = min(m + g, ldz - 1);
#pragma unroll
        for (int q = 0; q < CT; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h) acc[q][h] = Zs[(8 * q + 2 * t + h) * ldz + row];
#pragma unroll
        for (int u = 0; u < 16; ++u)
#pragma unroll
          for (int q = 0; q < CT; ++q) dmma(acc[q][0], acc[q][1], f[u], Ys[(8 * q + g) * XLD + 4 * u + t]);
#pragma unroll
        for (int q = 0; q < CT; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (m + g < n) Zs[(8 * q + 2 * t + h) * ldz + m + g] = acc[q][h];
#pragma unroll
        for (int u = 0; u < 16; ++u) f[u] = fn[u];
      }
    }
    __syncthreads();
  }
  for (int c = 0; c < NC; ++c)
    if (c0 + c < n)
      for (int i = tid; i < n; i += NT) P.Z[i + (size_t)(c0 + c) * n] = Zs[c * ldz + i];
}

// A slab takes at most half an SM's shared memory, so that one CTA's loads
// overlap another's products: blocks up to n = 1616 with 8 columns.  Measured
// (one block, 8 columns; three grouped GEMMs per 64 reflectors in brackets): n = 100
// 0.019 ms (0.126), 301 0.052 (0.351), 512 0.103 (0.575), 1024 0.366 (1.123),
// 1400 0.751 (1.612); with one CTA an SM 1776 2.20 (2.28), 2400 5.8 (3.8), where
// every slab's reading of V from L2 is the limit.
constexpr size_t SLAB_SMEM = 227 * 1024 / 2;
constexpr size_t WY_SMEM = 2 * (size_t)BT_NB * (BT_NB + 1) * sizeof(double);

}  // namespace

int bt_slab_nmax() {
  int n = 64;
  while (slab_smem(n + 16, 8) <= SLAB_SMEM) n += 16;
  return n;
}

// 16 columns halve the reading of V; they pay when they still give every SM
// work (2368 columns on 148 SMs).
int bt_slab_columns(long columns, int nmax) {
  return columns >= 16L * 148 && slab_smem(nmax, 16) <= SLAB_SMEM ? 16 : 8;
}

cudaError_t bt_wy_launch(const BtSlabProb* d, int nprob, int blocks, cudaStream_t st) {
  if (blocks <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(bt_wy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WY_SMEM);
  if (e != cudaSuccess) return e;
  NRGB_LAUNCH("bt_T", st, bt_wy_kernel<<<blocks, NT, WY_SMEM, st>>>(d, nprob));
  return cudaGetLastError();
}

cudaError_t bt_apply_launch(const BtSlabProb* d, int nprob, int columns, int ctas, int nmax, cudaStream_t st) {
  if (ctas <= 0) return cudaSuccess;
  // every caller sets the same value, so threads that race here agree
  cudaError_t e = columns == 16 ? cudaFuncSetAttribute(bt_apply_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SLAB_SMEM)
                                : cudaFuncSetAttribute(bt_apply_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SLAB_SMEM);
  if (e != cudaSuccess) return e;
  const size_t smem = slab_smem(nmax, columns);
  if (columns == 16) NRGB_LAUNCH("bt_apply", st, bt_apply_kernel<2><<<ctas, NT, smem, st>>>(d, nprob));
  else NRGB_LAUNCH("bt_apply", st, bt_apply_kernel<1><<<ctas, NT, smem, st>>>(d, nprob));
  return cudaGetLastError();
}

}  // namespace nrgb
