// Grouped, segmented-K FP64 GEMM on the DMMA tensor-core path (sm_100a).
// See gemm_f64.cuh for the contract.
//
// 64x64 tiles per CTA on 4 warps of 32x32 (32x32 tiles for launches with few
// of them), K staged 16 at a time through a cp.async ring laid out so that
// the DMMA fragment loads are bank-conflict free; 128x128 tiles where the
// schedule picks them.  mma.sync.m8n8k4.f64 (the m16n8k4/k8/k16 f64 shapes run
// at the same rate on B200): A fragment A[g][t], B fragment B[t][g], accumulator
// C[g][2t..2t+1] with g = lane/4, t = lane%4.
#include <string.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "common.cuh"
#include "gemm_f64.cuh"
#include "schedule.cuh"

namespace nrgb {

namespace {

constexpr int BM = GEMM_BM, BN = GEMM_BN, BK = GEMM_BK;
constexpr int NT = 128;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// Large-tile variant: 128x128 per CTA, 8 warps of 64x32, K staged 16 at a
// time through a 3-stage cp.async pipeline (8-byte copies with zero fill at
// the edges, so no register staging); the segment's alpha scales the A
// fragments after the shared-memory load.
// ---------------------------------------------------------------------------
constexpr int LBM = 128, LBN = 128, LSTAGES = 3, LNT = 256;
constexpr int LLDS = LBM + 4;  // 132: t*132+g -> distinct bank pairs

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__global__ void __launch_bounds__(LNT) gemm_grouped_large_kernel(const GemmProb* __restrict__ probs,
                                                                 int nprob,
                                                                 const GemmSeg* __restrict__ segs,
                                                                 const int* const* __restrict__ cmaps) {
  extern __shared__ __align__(16) double lsm[];
  double* As = lsm;                               // [LSTAGES][BK][LLDS]
  double* Bs = lsm + LSTAGES * BK * LLDS;         // [LSTAGES][BK][LLDS]
  __shared__ double salpha[LSTAGES];
  const int tile = blockIdx.x;
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].stile0 <= tile) lo = mid; else hi = mid - 1;
  }
  const GemmProb P = probs[lo];
  const int ks = P.ksplit > 1 ? P.ksplit : 1;
  const int t = (tile - P.stile0) / ks;
  const int kc = (tile - P.stile0) % ks;
  const int row0 = (t / P.stiles_n) * LBM;
  const int col0 = (t % P.stiles_n) * LBN;
  const int m = P.m, n = P.n;
  if (row0 >= m || col0 >= n) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tq = lane & 3;
  const int wm = (warp & 1) * 64, wn = (warp >> 1) * 32;

  double acc[8][4][2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int send = P.seg0 + P.nseg;
  int ktot = 0;
  for (int q = P.seg0; q < send; ++q) ktot += segs[q].k > 0 ? (segs[q].k + BK - 1) / BK : 0;
  const int per = (ktot + ks - 1) / ks;
  const int kt0 = kc * per;
  const int nk = max(0, min(ktot, kt0 + per) - kt0);
  // load cursor
  int ls = P.seg0, lk0 = 0;
  {
    int kt = 0;
    while (ls < send) {
      const int nt = segs[ls].k > 0 ? (segs[ls].k + BK - 1) / BK : 0;
      if (kt + nt > kt0) break;
      kt += nt;
      ++ls;
    }
    lk0 = (kt0 - kt) * BK;
  }
  auto issue = [&](int stage) {
    const GemmSeg S = segs[ls];
    double* as = As + stage * BK * LLDS;
    double* bs = Bs + stage * BK * LLDS;
    if (!S.transA) {
      const int i = tid & 127, pb = tid >> 7;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int p = pb + 2 * r, gi = row0 + i, gp = lk0 + p;
        const bool ok = gi < m && gp < S.k;
        cp_async8(&as[p * LLDS + i], ok ? S.A + (size_t)gp * S.lda + gi : S.A, ok);
      }
    } else {
      const int p = tid & 15, ib = tid >> 4;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int i = ib + 16 * r, gi = row0 + i, gp = lk0 + p;
        const bool ok = gi < m && gp < S.k;
        cp_async8(&as[p * LLDS + i], ok ? S.A + (size_t)gi * S.lda + gp : S.A, ok);
      }
    }
    if (!S.transB) {
      const int p = tid & 15, jb = tid >> 4;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int j = jb + 16 * r, gj = col0 + j, gp = lk0 + p;
        const bool ok = gj < n && gp < S.k;
        cp_async8(&bs[p * LLDS + j], ok ? S.B + (size_t)gj * S.ldb + gp : S.B, ok);
      }
    } else {
      const int j = tid & 127, pb = tid >> 7;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int p = pb + 2 * r, gj = col0 + j, gp = lk0 + p;
        const bool ok = gj < n && gp < S.k;
        cp_async8(&bs[p * LLDS + j], ok ? S.B + (size_t)gp * S.ldb + gj : S.B, ok);
      }
    }
    if (tid == 0) salpha[stage] = S.alpha;
    // advance the cursor
    lk0 += BK;
    if (lk0 >= S.k) {
      ++ls;
      while (ls < send && segs[ls].k <= 0) ++ls;
      lk0 = 0;
    }
  };
  // prologue
#pragma unroll
  for (int st = 0; st < LSTAGES - 1; ++st) {
    if (st < nk) issue(st);
    cp_async_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<LSTAGES - 2>();
    __syncthreads();
    const int nxt = kt + LSTAGES - 1;
    if (nxt < nk) issue(nxt % LSTAGES);
    cp_async_commit();
    const int stg = kt % LSTAGES;
    const double* as = As + stg * BK * LLDS;
    const double* bs = Bs + stg * BK * LLDS;
    const double alpha = salpha[stg];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      double a[8], b[4];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = alpha * as[(kk + tq) * LLDS + wm + i * 8 + g];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = bs[(kk + tq) * LLDS + wn + j * 8 + g];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  cp_async_wait<0>();
  const double beta = P.beta;
  const int* cmap = cmaps ? cmaps[lo] : nullptr;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row0 + wm + i * 8 + g;
    if (r >= m) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = col0 + wn + j * 8 + 2 * tq + h;
        if (c < n) {
          double* dst = P.C + (size_t)(cmap ? cmap[c] : c) * P.ldc + r;
          const double v = acc[i][j][h];
          if (ks > 1) atomicAdd(dst, v);
          else *dst = (beta == 0.0) ? v : v + beta * (*dst);
        }
      }
    }
  }
}

constexpr size_t LSMEM = 2 * (size_t)LSTAGES * BK * LLDS * sizeof(double);

// ---------------------------------------------------------------------------
// Pipelined kernel: T x T tiles (64 or 32) on 4 warps of T/2 x T/2, operands
// copied by cp.async into a ring of three K steps of 16.  Each operand tile
// keeps the direction in which it is contiguous in global memory:
//   mn-contiguous (A as stored, B transposed): [16][T + 4]
//   k-contiguous  (A transposed, B as stored): [T][16], the 16-byte pairs of
//     row r at pair index (p/2) ^ (2r mod 8)
// and both are read bank-conflict free by the fragment loads (within a
// half-warp, lanes g, t hit double offsets 4t + g, resp. 2((k/2 + t/2) ^ 2g)
// + t%2, mod 16, all distinct).  A segment whose base address and leading
// dimension are 16-byte aligned is copied in element pairs (16-byte cp.async;
// the half of a pair outside the matrix is zero-filled), any other segment
// (sub-blocks of eigenvector matrices mostly) element by element.
//
// What bounds it is the FP64 tensor pipe (16 cycles an m8n8k4) and the issue
// slots around it, so everything that does not change from K step to K step
// (source pointers, strides, row bounds, the swizzled offsets) stays in
// registers: nine instructions went with every tensor instruction when each
// step derived them from the segment again.  A CTA finds its problem with one
// or two loads by all lanes (a binary search was a chain of up to ten), and
// small launches get their descriptors as kernel parameters instead of copies.
// ---------------------------------------------------------------------------
constexpr int KB = BK, STAGES = 3;

template <int T>
__host__ __device__ constexpr int ptile() { return KB * (T + 4); }

__device__ __forceinline__ void cp_async16(double* smem, const double* gmem, int bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

// One operand's copies of a thread: a T x 16 tile of a matrix whose element
// (mn, k) sits at base[mn + k ld] (mn-contiguous) or base[k + mn ld].
template <int T>
struct Operand {
  const double* p;  // the thread's first element of the next K step
  int ld, lim;      // leading dimension; rows of the tile inside the matrix
  int mode;         // bit 0: pairs, bit 1: k-contiguous

  __device__ __forceinline__ void set(const double* base, int ld_, bool kcont, int mn0, int mnlim, int k0, int tid) {
    ld = ld_;
    lim = mnlim - mn0;
    const bool vec = ((reinterpret_cast<uintptr_t>(base) & 15) == 0) && ((ld & 1) == 0);
    mode = (vec ? 1 : 0) | (kcont ? 2 : 0);
    int i, k;
    if (mode == 0) {
      i = tid & (T - 1);
      k = tid / T;
    } else if (mode == 1) {
      i = 2 * (tid & (T / 2 - 1));
      k = tid / (T / 2);
    } else if (mode == 2) {
      i = tid >> 4;
      k = tid & 15;
    } else {
      i = tid >> 3;
      k = 2 * (tid & 7);
    }
    p = base + (kcont ? (size_t)(mn0 + i) * ld + (k0 + k) : (size_t)(k0 + k) * ld + (mn0 + i));
  }
  // Copies the tile (krem columns are inside the matrix) and steps on.
  __device__ __forceinline__ void issue(double* dst, int krem, int tid) {
    if (mode == 0) {
      const int i = tid & (T - 1), k = tid / T;
      const size_t step = (size_t)(NT / T) * ld;
      const bool in = i < lim;
      const double* q = p;
#pragma unroll
      for (int r = 0; r < KB * T / NT; ++r) {
        cp_async8(dst + (k + NT / T * r) * (T + 4) + i, q, in && k + NT / T * r < krem);
        q += step;
      }
    } else if (mode == 1) {
      const int i = 2 * (tid & (T / 2 - 1)), k = tid / (T / 2);
      const size_t step = (size_t)(2 * NT / T) * ld;
      const int bytes = min(max(lim - i, 0), 2) * 8;
      const double* q = p;
#pragma unroll
      for (int r = 0; r < KB * T / (2 * NT); ++r) {
        cp_async16(dst + (k + 2 * NT / T * r) * (T + 4) + i, q, k + 2 * NT / T * r < krem ? bytes : 0);
        q += step;
      }
    } else if (mode == 2) {
      const int i = tid >> 4, k = tid & 15;
      const size_t step = (size_t)8 * ld;
      double* d = dst + i * KB + (((k >> 1) ^ ((2 * i) & 7)) << 1) + (k & 1);
      const int rows = k < krem ? lim - i : 0;
      const double* q = p;
#pragma unroll
      for (int r = 0; r < T / 8; ++r) {
        cp_async8(d + 8 * KB * r, q, 8 * r < rows);
        q += step;
      }
    } else {
      const int i = tid >> 3, k = 2 * (tid & 7);
      const size_t step = (size_t)16 * ld;
      double* d = dst + i * KB + (((k >> 1) ^ ((2 * i) & 7)) << 1);
      const int bytes = min(max(krem - k, 0), 2) * 8, rows = lim - i;
      const double* q = p;
#pragma unroll
      for (int r = 0; r < T / 16; ++r) {
        cp_async16(d + 16 * KB * r, q, 16 * r < rows ? bytes : 0);
        q += step;
      }
    }
    p += (mode & 2) ? (size_t)KB : (size_t)KB * ld;
  }
};

// The products of one K step; FL: bit 0 A k-contiguous, bit 1 B k-contiguous;
// SC: A is scaled by alpha.  (A test of alpha between the loads and the products
// kept the compiler from loading ahead: 29.5 TF/s on 37 products of edge 1024,
// 32.5 without scaling, 29.2 with.)
template <int T, bool SC, int FL>
__device__ __forceinline__ void tile_step(double (&acc)[T / 16][T / 16][2], const double* as, const double* bs,
                                          double alpha, int wm, int wn, int g, int tq, const int (&ko)[4]) {
  constexpr int W = T / 16;
  const double* ap = (FL & 1) ? as + (wm + g) * KB : as + tq * (T + 4) + wm + g;
  const double* bp = (FL & 2) ? bs + (wn + g) * KB : bs + tq * (T + 4) + wn + g;
#pragma unroll
  for (int kk = 0; kk < KB; kk += 4) {
    double a[W], b[W];
#pragma unroll
    for (int i = 0; i < W; ++i) a[i] = (FL & 1) ? ap[ko[kk / 4] + i * 8 * KB] : ap[kk * (T + 4) + i * 8];
#pragma unroll
    for (int j = 0; j < W; ++j) b[j] = (FL & 2) ? bp[ko[kk / 4] + j * 8 * KB] : bp[kk * (T + 4) + j * 8];
    if constexpr (SC) {
#pragma unroll
      for (int i = 0; i < W; ++i) a[i] *= alpha;
    }
#pragma unroll
    for (int i = 0; i < W; ++i)
#pragma unroll
      for (int q = 0; q < W; ++q) {
        const int j = (i & 1) ? W - 1 - q : q;  // back and forth: one fragment stays
        dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
      }
  }
}

// Last problem whose tile0 is at most `tile` (all lanes of a warp call it).
__device__ __forceinline__ int find_problem(const GemmProb* probs, int nprob, int tile, int lane) {
  int lo = 0, len = nprob;
  while (len > 1) {
    const int step = (len + 31) / 32, i = lo + lane * step;
    const bool le = lane * step < len && (lane == 0 || probs[i].tile0 <= tile);
    const int last = 31 - __clz(__ballot_sync(0xffffffffu, le));
    lo += last * step;
    len = min(step, len - last * step);
  }
  return lo;
}

template <int T, bool SC>
__device__ __forceinline__ void gemm_tile(const GemmProb* __restrict__ probs, int nprob, const GemmSeg* __restrict__ segs,
                                          const int* const* __restrict__ cmaps) {
  constexpr int W = T / 16, PT = ptile<T>(), SUB = 64 / T;  // SUB^2 CTAs share a 64 x 64 tile
  extern __shared__ __align__(16) double psm[];
  double* As = psm;                 // [STAGES][PT]
  double* Bs = psm + STAGES * PT;   // [STAGES][PT]
  __shared__ double salpha[STAGES];
  __shared__ int sflags[STAGES];    // see tile_step

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = blockIdx.x / (SUB * SUB), sub = blockIdx.x % (SUB * SUB);
  const int lo = find_problem(probs, nprob, tile, lane);
  const GemmProb P = probs[lo];
  const int ks = P.ksplit > 1 ? P.ksplit : 1;
  const int t = (tile - P.tile0) / ks;
  const int kc = (tile - P.tile0) % ks;
  const int row0 = (t / P.tiles_n) * BM + (sub / SUB) * T;
  const int col0 = (t % P.tiles_n) * BN + (sub % SUB) * T;
  const int m = P.m, n = P.n;
  if (row0 >= m || col0 >= n) return;  // also shapes set on the device below the planned bound

  const int g = lane >> 2, tq = lane & 3;
  const int wm = (warp & 1) * (T / 2), wn = (warp >> 1) * (T / 2);
  int ko[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) ko[q] = (((2 * q + (tq >> 1)) ^ ((2 * g) & 7)) << 1) + (tq & 1);

  double acc[W][W][2];
#pragma unroll
  for (int i = 0; i < W; ++i)
#pragma unroll
    for (int j = 0; j < W; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  // this CTA's share of the flattened (segment, K step) sequence
  const int send = P.seg0 + P.nseg;
  int ktot = 0;
  for (int q = P.seg0 + lane; q < send; q += 32) ktot += segs[q].k > 0 ? (segs[q].k + KB - 1) / KB : 0;
  ktot = __reduce_add_sync(0xffffffffu, ktot);
  const int per = (ktot + ks - 1) / ks;
  const int kt0 = kc * per;
  const int nk = max(0, min(ktot, kt0 + per) - kt0);
  int ls = P.seg0, kleft = 0;  // current segment, its K columns not yet copied
  Operand<T> oa, ob;
  double alpha_l = 1.0;
  auto open = [&](int k0) {
    const GemmSeg G = segs[ls];
    // op(A)[i, p]: A[i + p lda] as stored, A[p + i lda] transposed
    oa.set(G.A, G.lda, G.transA != 0, row0, m, k0, tid);
    // op(B)[p, j]: B[p + j ldb] as stored (k-contiguous), B[j + p ldb] transposed
    ob.set(G.B, G.ldb, G.transB == 0, col0, n, k0, tid);
    alpha_l = G.alpha;
    kleft = G.k - k0;
  };
  if (nk > 0) {
    int kt = 0;
    while (true) {
      const int k = segs[ls].k, nt = k > 0 ? (k + KB - 1) / KB : 0;
      if (kt + nt > kt0) break;
      kt += nt;
      ++ls;
    }
    open((kt0 - kt) * KB);
  }
  auto issue = [&](int stage) {
    if (kleft <= 0) {
      do ++ls;
      while (segs[ls].k <= 0);
      open(0);
    }
    oa.issue(As + stage * PT, kleft, tid);
    ob.issue(Bs + stage * PT, kleft, tid);
    kleft -= KB;
    if (tid == 0) {
      salpha[stage] = alpha_l;
      sflags[stage] = (oa.mode >> 1) | (ob.mode & 2);
    }
  };
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < nk) issue(st);
    cp_async_commit();
  }
  int stg = 0, nxt = STAGES - 1;
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (kt + STAGES - 1 < nk) issue(nxt);
    cp_async_commit();
    const double* as = As + stg * PT;
    const double* bs = Bs + stg * PT;
    const double alpha = salpha[stg];
    switch (sflags[stg]) {
      case 0: tile_step<T, SC, 0>(acc, as, bs, alpha, wm, wn, g, tq, ko); break;
      case 1: tile_step<T, SC, 1>(acc, as, bs, alpha, wm, wn, g, tq, ko); break;
      case 2: tile_step<T, SC, 2>(acc, as, bs, alpha, wm, wn, g, tq, ko); break;
      default: tile_step<T, SC, 3>(acc, as, bs, alpha, wm, wn, g, tq, ko); break;
    }
    stg = stg + 1 == STAGES ? 0 : stg + 1;
    nxt = nxt + 1 == STAGES ? 0 : nxt + 1;
  }
  cp_async_wait<0>();

  // With beta the loads of a row of fragments come before its stores: one after
  // the other, each behind the store before it, they cost 32 trips a tile (57
  // trailing updates with K = 64: 5.7 ms, 3.9 now).
  const double beta = P.beta;
  const int* cmap = cmaps ? cmaps[lo] : nullptr;
  const bool rmw = ks == 1 && beta != 0.0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const int r = row0 + wm + i * 8 + g;
    if (r >= m) continue;
    if (rmw) {
#pragma unroll
      for (int q = 0; q < 2 * W; ++q) {
        const int c = col0 + wn + (q >> 1) * 8 + 2 * tq + (q & 1);
        const double old = c < n ? P.C[(size_t)(cmap ? cmap[c] : c) * P.ldc + r] : 0.0;
        acc[i][q >> 1][q & 1] += beta * old;
      }
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = col0 + wn + j * 8 + 2 * tq + h;
        if (c < n) {
          double* dst = P.C + (size_t)(cmap ? cmap[c] : c) * P.ldc + r;
          if (ks > 1) atomicAdd(dst, acc[i][j][h]);
          else *dst = acc[i][j][h];
        }
      }
    }
  }
}

// 128 registers at most, so that shared memory alone sets the CTAs per SM
// (52 KB each with T = 64: four).  SC: some segment's alpha is not one.
template <int T, bool SC>
__global__ void __launch_bounds__(NT, T == 64 ? 4 : 6) gemm_grouped_pipe_kernel(const GemmProb* __restrict__ probs, int nprob,
                                                                  const GemmSeg* __restrict__ segs,
                                                                  const int* const* __restrict__ cmaps) {
  gemm_tile<T, SC>(probs, nprob, segs, cmaps);
}

// The descriptors of a small launch as a kernel parameter: problems, then segments.
template <int BYTES>
struct InlineDesc {
  alignas(16) unsigned char b[BYTES];
};
template <int T, bool SC, int BYTES>
__global__ void __launch_bounds__(NT, T == 64 ? 4 : 6) gemm_grouped_inline_kernel(const __grid_constant__ InlineDesc<BYTES> d,
                                                                    int nprob) {
  const GemmProb* probs = reinterpret_cast<const GemmProb*>(d.b);
  gemm_tile<T, SC>(probs, nprob, reinterpret_cast<const GemmSeg*>(probs + nprob), nullptr);
}

template <int T>
constexpr size_t pipe_smem() { return 2 * (size_t)STAGES * ptile<T>() * sizeof(double); }

// Dynamic shared memory of the kernels above, once per device (every caller
// sets the same values, so threads that race here agree).
cudaError_t pipe_attributes() {
  static std::atomic<bool> set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && set[dev].load(std::memory_order_acquire)) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  auto one = [&](auto* k, size_t bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  auto both = [&](auto* plain, auto* scaled, size_t bytes) {
    one(plain, bytes);
    one(scaled, bytes);
  };
  both(gemm_grouped_pipe_kernel<64, false>, gemm_grouped_pipe_kernel<64, true>, pipe_smem<64>());
  both(gemm_grouped_pipe_kernel<32, false>, gemm_grouped_pipe_kernel<32, true>, pipe_smem<32>());
  both(gemm_grouped_inline_kernel<64, false, 4096>, gemm_grouped_inline_kernel<64, true, 4096>, pipe_smem<64>());
  both(gemm_grouped_inline_kernel<32, false, 4096>, gemm_grouped_inline_kernel<32, true, 4096>, pipe_smem<32>());
  both(gemm_grouped_inline_kernel<64, false, 8192>, gemm_grouped_inline_kernel<64, true, 8192>, pipe_smem<64>());
  both(gemm_grouped_inline_kernel<32, false, 8192>, gemm_grouped_inline_kernel<32, true, 8192>, pipe_smem<32>());
  both(gemm_grouped_inline_kernel<64, false, 16384>, gemm_grouped_inline_kernel<64, true, 16384>, pipe_smem<64>());
  both(gemm_grouped_inline_kernel<32, false, 16384>, gemm_grouped_inline_kernel<32, true, 16384>, pipe_smem<32>());
  both(gemm_grouped_inline_kernel<64, false, GEMM_INLINE_MAX>, gemm_grouped_inline_kernel<64, true, GEMM_INLINE_MAX>,
       pipe_smem<64>());
  both(gemm_grouped_inline_kernel<32, false, GEMM_INLINE_MAX>, gemm_grouped_inline_kernel<32, true, GEMM_INLINE_MAX>,
       pipe_smem<32>());
  if (e == cudaSuccess && dev < 64) set[dev].store(true, std::memory_order_release);
  return e;
}

// Tile edge of a launch: four 32 x 32 CTAs for each 64 x 64 tile where those
// would leave SMs idle, or where the problems are small (60 tiles: an edge of
// 480) and at least 3 % of the 64 x 64 tiles' area lies outside them in quarters
// that 32 x 32 tiles leave out, so that the rims outweigh the operands read twice
// as often (12 % more time for the same area), or the SMs with one tile more than
// the others would cost more than that.  Measured (64 / 32, us; area that is left out): one 500^3 44.8 / 29.1
// (idle SMs), four 300^3 32.4 / 26.0 (idle SMs), eight of 200-300 34.8 / 29.6 (14 %),
// twelve of 400-500 120.5 / 105.8 (7 %), eighty of 100-300 84.0 / 83.9 (13 %), eight
// 384^3 44.8 / 50.8 (none), forty 512^3 358.8 / 405.3 (none), two 700^3 70.6 / 80.9
// (none), sixteen 448^3 156 / 166 (none; 13 % lost to the last tiles), forty products
// of 256^3 134 / 119 (none; 16 %).  Within 5 % either way, by how the last wave falls: eight of 300-400 45.7 /
// 46.1 (4 %), sixteen of them 75.8 / 78.2 (6 %), forty of 200-400 112.8 / 117.9 (9 %).
bool use_small_tiles(int total_tiles, int nprob, int tiles32) {
  if (total_tiles < 148) return true;
  if (total_tiles > 60L * nprob) return false;
  const long busiest = (total_tiles + 147) / 148;  // tiles of the SM with the most
  return tiles32 <= 3.88 * total_tiles || 148 * busiest > 1.15 * total_tiles;
}

// Order of the problems of a launch described on the host: those whose tiles
// have the most K steps first where the launch takes more than one wave of CTAs
// (six per SM with T = 32, four with 64), so that the last wave ends with short
// tiles.  64 outputs of four terms (K 15 to 115 each), 3544 CTAs: 112.9 us in the
// caller's order, 105.1 sorted.  In 64 classes of steps, in time linear in the
// problems (a comparison sort and a copy of descriptors that stayed as they were
// took 15 to 20 us of host time for a thousand problems, more than it gave);
// problems of one class keep their order.
struct ProblemOrder {
  static constexpr int CLASSES = 64;
  int at[CLASSES + 1] = {};  // first place of a class, the longest first

  // The problems' classes in key; false: the caller's order stands.
  bool classes(const GemmProb* probs, int nprob, const GemmSeg* segs, int total_tiles, bool small, int* key) {
    if (nprob == 1 || (small ? 4L : 1L) * total_tiles <= (small ? 6L : 4L) * 148) return false;
    int most = 0;
    for (int p = 0; p < nprob; ++p) {
      long steps = 0;
      for (int q = probs[p].seg0; q < probs[p].seg0 + probs[p].nseg; ++q)
        if (segs[q].k > 0) steps += (segs[q].k + KB - 1) / KB;
      key[p] = (int)std::min(steps / std::max(1, probs[p].ksplit), 0x7fffffffL);
      most = std::max(most, key[p]);
    }
    const double scale = (CLASSES - 1) / std::max(1.0, (double)most);
    bool ordered = true;
    for (int p = 0; p < nprob; ++p) {
      key[p] = CLASSES - 1 - (int)(key[p] * scale);
      ++at[key[p] + 1];
      ordered = ordered && (p == 0 || key[p - 1] <= key[p]);
    }
    return !ordered;
  }
  void copy(const GemmProb* probs, int nprob, const int* key, GemmProb* out) {
    for (int c = 0; c < CLASSES; ++c) at[c + 1] += at[c];
    for (int p = 0; p < nprob; ++p) out[at[key[p]]++] = probs[p];
    int tiles = 0, stiles = 0;
    for (int i = 0; i < nprob; ++i) gemm_assign_tiles(out[i], tiles, stiles);
  }
};

cudaError_t pipe_launch(const GemmProb* d_probs, int nprob, const GemmSeg* d_segs, int total_tiles, int tiles32,
                        cudaStream_t stream, const int* const* cmaps, bool scaled) {
  const cudaError_t e = pipe_attributes();
  if (e != cudaSuccess) return e;
  const bool small = use_small_tiles(total_tiles, nprob, tiles32);
  const auto k = small ? (scaled ? gemm_grouped_pipe_kernel<32, true> : gemm_grouped_pipe_kernel<32, false>)
                       : (scaled ? gemm_grouped_pipe_kernel<64, true> : gemm_grouped_pipe_kernel<64, false>);
  k<<<(small ? 4 : 1) * total_tiles, NT, small ? pipe_smem<32>() : pipe_smem<64>(), stream>>>(d_probs, nprob, d_segs, cmaps);
  return cudaGetLastError();
}

template <int BYTES>
cudaError_t inline_launch(const GemmProb* probs, int nprob, const GemmSeg* segs, int nseg, int total_tiles,
                          cudaStream_t stream) {
  InlineDesc<BYTES> d;
  const bool small = use_small_tiles(total_tiles, nprob, gemm_tiles32(probs, nprob)), scaled = gemm_scaled(segs, nseg);
  ProblemOrder order;
  int key[GEMM_INLINE_MAX / sizeof(GemmProb)];
  if (order.classes(probs, nprob, segs, total_tiles, small, key)) order.copy(probs, nprob, key, reinterpret_cast<GemmProb*>(d.b));
  else memcpy(d.b, probs, nprob * sizeof(GemmProb));
  memcpy(d.b + nprob * sizeof(GemmProb), segs, nseg * sizeof(GemmSeg));
  const auto k = small ? (scaled ? gemm_grouped_inline_kernel<32, true, BYTES> : gemm_grouped_inline_kernel<32, false, BYTES>)
                       : (scaled ? gemm_grouped_inline_kernel<64, true, BYTES> : gemm_grouped_inline_kernel<64, false, BYTES>);
  k<<<(small ? 4 : 1) * total_tiles, NT, small ? pipe_smem<32>() : pipe_smem<64>(), stream>>>(d, nprob);
  return cudaGetLastError();
}

// The 128x128 cp.async variant is used only where the device's schedule
// (schedule.cuh, set by the autotuner's measurements) says it wins: by
// default never (the autotuner's launches on B200: 21-24 TF/s at edges of 256 to
// 2048 against 28-29 TF/s for the tiles above; 27.8 against 27.6 at 192, which
// is within its margin).

}  // namespace

void gemm_assign_tiles(GemmProb& p, int& tiles, int& stiles) {
  const int ks = p.ksplit > 1 ? p.ksplit : 1;
  p.tile0 = tiles;
  p.tiles_n = (p.n + GEMM_BN - 1) / GEMM_BN;
  tiles += ((p.m + GEMM_BM - 1) / GEMM_BM) * p.tiles_n * ks;
  p.stile0 = stiles;
  p.stiles_n = (p.n + LBN - 1) / LBN;
  stiles += ((p.m + LBM - 1) / LBM) * p.stiles_n * ks;
}

int gemm_tiles32(const GemmProb* probs, int nprob) {
  int t = 0;
  for (int p = 0; p < nprob; ++p)
    t += ((probs[p].m + 31) / 32) * ((probs[p].n + 31) / 32) * (probs[p].ksplit > 1 ? probs[p].ksplit : 1);
  return t;
}

bool gemm_scaled(const GemmSeg* segs, int nseg) {
  for (int s = 0; s < nseg; ++s)
    if (segs[s].alpha != 1.0) return true;
  return false;
}

double gemm_flops(const GemmProb* probs, int nprob, const GemmSeg* segs) {
  double f = 0;
  for (int p = 0; p < nprob; ++p)
    for (int s = probs[p].seg0; s < probs[p].seg0 + probs[p].nseg; ++s)
      f += 2.0 * probs[p].m * (double)probs[p].n * segs[s].k;
  return f;
}

cudaError_t gemm_grouped_launch(const GemmProb* d_probs, int nprob, const GemmSeg* d_segs,
                                int total_tiles, cudaStream_t stream, const char* tag, int tiles32, int total_stiles,
                                const int* const* cmaps, bool scaled) {
  if (total_tiles <= 0 || nprob <= 0) return cudaSuccess;
  // 128x128 tiles when the schedule selects them for this problem size,
  // they cover at most 30% more area than the 64x64 ones and they still give
  // enough CTAs to fill the GPU
  const int large_from = schedule_here().gemm_large_from.load(std::memory_order_relaxed);
  const double edge = GEMM_BM * sqrt((double)total_tiles / nprob);  // mean output edge per problem
  if (large_from > 0 && edge >= large_from && total_stiles > 0 && 4.0 * total_stiles <= 1.3 * total_tiles &&
      total_stiles >= 120) {
    // once per device (function attributes belong to the device's context);
    // every caller sets the same value, so threads that race here agree
    static std::atomic<bool> attr[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
      const cudaError_t e =
          cudaFuncSetAttribute(gemm_grouped_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LSMEM);
      if (e != cudaSuccess) return e;
      if (dev < 64) attr[dev].store(true, std::memory_order_release);
    }
    NRGB_LAUNCH(tag, stream,
                gemm_grouped_large_kernel<<<total_stiles, LNT, LSMEM, stream>>>(d_probs, nprob, d_segs, cmaps));
    return cudaGetLastError();
  }
  cudaError_t e = cudaSuccess;
  NRGB_LAUNCH(tag, stream, e = pipe_launch(d_probs, nprob, d_segs, total_tiles, tiles32, stream, cmaps, scaled));
  return e;
}

cudaError_t gemm_grouped_launch_unaccounted(const GemmProb* d_probs, int nprob, const GemmSeg* d_segs,
                                            int total_tiles, int tiles32, cudaStream_t stream, bool scaled) {
  if (total_tiles <= 0 || nprob <= 0) return cudaSuccess;
  return pipe_launch(d_probs, nprob, d_segs, total_tiles, tiles32, stream, nullptr, scaled);
}

size_t gemm_desc_bytes(int nprob, int nseg) {
  return nprob * sizeof(GemmProb) + nseg * sizeof(GemmSeg) + 1024;
}

cudaError_t gemm_grouped_launch_host(const GemmProb* probs, int nprob, const GemmSeg* segs, int nseg, int total_tiles,
                                     cudaStream_t stream, const char* tag, int total_stiles, const GemmStage& stage) {
  if (total_tiles <= 0 || nprob <= 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (gemm_inline_fits(nprob, nseg) && schedule_here().gemm_large_from.load(std::memory_order_relaxed) == 0) {
    NRGB_LAUNCH(tag, stream, e = gemm_grouped_launch_inline(probs, nprob, segs, nseg, total_tiles, stream));
    return e;
  }
  const int tiles32 = gemm_tiles32(probs, nprob);
  ProblemOrder order;
  std::vector<GemmProb> ordered;
  std::vector<int> key(nprob);
  if (order.classes(probs, nprob, segs, total_tiles, use_small_tiles(total_tiles, nprob, tiles32), key.data())) {
    ordered.resize(nprob);
    order.copy(probs, nprob, key.data(), ordered.data());
    probs = ordered.data();
  }
  const GemmProb* dp = static_cast<const GemmProb*>(stage(probs, nprob * sizeof(GemmProb)));
  const GemmSeg* ds = static_cast<const GemmSeg*>(stage(segs, nseg * sizeof(GemmSeg)));
  return gemm_grouped_launch(dp, nprob, ds, total_tiles, stream, tag, tiles32, total_stiles, nullptr,
                             gemm_scaled(segs, nseg));
}

cudaError_t gemm_grouped_launch_host(const GemmProb* probs, int nprob, const GemmSeg* segs, int nseg, int total_tiles,
                                     cudaStream_t stream, const char* tag, int total_stiles, DeviceArena& scratch) {
  return gemm_grouped_launch_host(probs, nprob, segs, nseg, total_tiles, stream, tag, total_stiles,
                                  [&](const void* src, size_t bytes) -> const void* {
                                    void* d = scratch.alloc(bytes);
                                    NRGB_CUDA(cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, stream));
                                    return d;
                                  });
}

bool gemm_inline_fits(int nprob, int nseg) {
  return nprob * sizeof(GemmProb) + nseg * sizeof(GemmSeg) <= (size_t)GEMM_INLINE_MAX;
}

// (a launch copies the whole parameter: four sizes of it; an allocation-free basis
// change of 40 operators, 4.2 KB twice, 39.0 us with 32000 bytes, 34.8 with 8192)
cudaError_t gemm_grouped_launch_inline(const GemmProb* probs, int nprob, const GemmSeg* segs, int nseg,
                                       int total_tiles, cudaStream_t stream) {
  if (total_tiles <= 0 || nprob <= 0) return cudaSuccess;
  const cudaError_t e = pipe_attributes();
  if (e != cudaSuccess) return e;
  if (nprob * sizeof(GemmProb) + nseg * sizeof(GemmSeg) <= 4096)
    return inline_launch<4096>(probs, nprob, segs, nseg, total_tiles, stream);
  if (nprob * sizeof(GemmProb) + nseg * sizeof(GemmSeg) <= 8192)
    return inline_launch<8192>(probs, nprob, segs, nseg, total_tiles, stream);
  if (nprob * sizeof(GemmProb) + nseg * sizeof(GemmSeg) <= 16384)
    return inline_launch<16384>(probs, nprob, segs, nseg, total_tiles, stream);
  return inline_launch<GEMM_INLINE_MAX>(probs, nprob, segs, nseg, total_tiles, stream);
}

}  // namespace nrgb
