// Batched FP64 symmetric eigensolver (see syev.cuh).
//
// Numerical methods (written from the published algorithms):
//  * Householder reflector H = I - tau v v^T, v(0) = 1, chosen so that
//    H x = beta e_1, beta = -sign(x_0) ||x||, tau = (beta - x_0)/beta.
//  * Blocked tridiagonalisation with the panel formulation A22 <- A22 - V W^T
//    - W V^T (Dongarra, Sorensen, Hammarling 1989).
//  * Divide and conquer: Cuppen's rank-one tearing, deflation of small z_i
//    and of close d_i by Givens rotations, secular-equation roots by a
//    safeguarded two-pole rational iteration (Bunch-Nielsen-Sorensen / Li
//    "middle way" model) in coordinates relative to the nearer pole, and
//    eigenvectors from the Loewner-formula z-hat (Gu & Eisenstat 1995), which
//    keeps them orthogonal without extra precision.
#include <map>
#include <mutex>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <numeric>

#include "bt_apply.cuh"
#include "dc_base.cuh"
#include "dc_secular.cuh"
#include "gemm_f64.cuh"
#include "reflector.cuh"
#include "syev.cuh"
#include "schedule.cuh"
#include "trd_grid.cuh"
#include "trd_regs.cuh"

namespace nrgb {

namespace {

constexpr int SMALL_N = SYEV_TINY;  // blocks solved whole in one CTA
constexpr int LEAF = DC_BASE;   // subtrees solved in one CTA (dc_base.cu)
constexpr int NB = 32;          // tridiagonalisation panel width
constexpr int TRAIL_STRIP = 256;  // columns of a strip of the trailing update
constexpr int NBB = BT_NB;      // back-transformation block of reflectors
constexpr int TRD_NT = 512;     // threads of the panel kernel, one CTA per SM
constexpr double EPS = 2.220446049250313e-16;

// --------------------------------------------------------------------------
// Tridiagonalisation panel (cooperative persistent kernel).
// --------------------------------------------------------------------------
struct TrdProb {
  double* A;    // n x n, ld n
  double* d;    // n
  double* e;    // n-1
  double* tau;  // n-1
  double* Vp;   // n x NB panel reflectors, row-major (row i at Vp + i*NB)
  double* W;    // n x NB, row-major
  double* y;    // slots of A22 v: see SymvShape
  double* red;  // 2 slots x (2 + 2*NB)
  GridBarrier* bar;  // this problem's barrier: only its own CTAs synchronise
  int n;
  int cta0, ncta;
  int wait_log2;     // a barrier wait gives up after 2^wait_log2 polls
  int expect_extra;  // CTAs the barriers expect beyond ncta (0; 1 injects a lost CTA)
};

constexpr int RED = 2 + 2 * NB;

__device__ __forceinline__ double ld_volatile(const double* p) {
  return *reinterpret_cast<const volatile double*>(p);
}

// Tiles of the product A22 v: 64 rows x 32 columns, one warp each, anchored at the
// panel's first row and column (base = j0 + 1; columns that the panel has finished
// meet zeros of v).  A tile on or below the diagonal gives its row sums to slot J
// of yr and the sums over its rows, of the elements below the diagonal, to slot I
// of yc: y_i = sum_{J <= i/32} yr[J][i] + sum_{I >= i/64} yc[I][i].
constexpr int SY_M = 64, SY_N = 32;
constexpr int TRD_SMEM = 32 + 4 * NB + 8 + (TRD_NT / 32) * 2 * NB;  // doubles before v

struct SymvShape {
  int M, nbm, nbn, mp;  // rows; blocks of 64 and of 32; padded rows
  __host__ __device__ explicit SymvShape(int rows)
      : M(rows), nbm((rows + SY_M - 1) / SY_M), nbn((rows + SY_N - 1) / SY_N), mp(nbm * SY_M) {}
};

// y_i (relative row) from every step-th of its slots, from the g-th on (yc lies
// behind yr, so that a slot is a multiple of mp away).
__device__ __forceinline__ double symv_sum(const SymvShape& S, const double* yr, int i, int g, int step) {
  const int nr = i / SY_N + 1, count = nr + S.nbm - i / SY_M, skip = S.nbn + i / SY_M - nr;
  double s = 0.0;
  for (int k = g; k < count; k += 16 * step) {
    double x[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int q = k + u * step;
      x[u] = q < count ? __ldcg(&yr[(size_t)(q < nr ? q : q + skip) * S.mp + i]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) s += x[u];
  }
  return s;
}

// d (8 x 8) += a (8 x 4) b (4 x 8), one warp; a lane holds a[lane / 4][lane % 4],
// b[lane % 4][lane / 4] and d[lane / 4][2 (lane % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// A warp's walk through its tiles, 8 columns at a time, with the elements of the
// next 8 in registers: a lane holds rows lane and 32 + lane of the tile.  Column
// blocks 2 s and 2 s + 1 have nbm - s tiles; blocks s and nbm - 1 - s together
// nbm + 1, so tile numbers decode with one division.
struct SymvWalk {
  const double* A;  // relative (0, 0)
  size_t ld;
  int M, nbm, nbn;
  int t, step;      // tile number
  int I, J, strip;  // where the elements in x are
  double x[16];

  __device__ __forceinline__ bool live() const { return I >= 0; }
  __device__ __forceinline__ int row() const { return I * SY_M + (threadIdx.x & 31); }
  __device__ __forceinline__ int col() const { return J * SY_N + 8 * strip; }
  // every column of the strip lies below the diagonal (and so within the matrix,
  // the tile's first row being one)
  __device__ __forceinline__ bool below() const { return col() + 7 < I * SY_M; }
  // the first tile from number t on
  __device__ __forceinline__ void settle() {
    const int folds = (nbm + 1) / 2;
    I = -1;
    for (; t < 2 * folds * (nbm + 1); t += step) {
      const int q = t >> 1, f = q / (nbm + 1), k = q - f * (nbm + 1);
      const bool first = k < nbm - f;
      const int s = first ? f : nbm - 1 - f;
      if (!first && s == f) continue;  // the middle block, counted once
      J = 2 * s + (t & 1);
      if (J >= nbn) continue;
      I = s + (first ? k : k - (nbm - f));
      break;
    }
    strip = 0;
  }
  __device__ __forceinline__ void advance() { skip(1); }
  __device__ __forceinline__ void skip(int strips) {  // up to the end of the tile
    strip += strips;
    if (strip == SY_N / 8) {
      t += step;
      settle();
    }
  }
  // Below the diagonal rows beyond the last are read as they come: at least eight
  // columns of the matrix follow, their v is zero and nobody reads their sums.
  __device__ __forceinline__ void load() {
    const int r = row(), c = col();
    const double* a = A + (r + c * ld);
    if (below()) {
#pragma unroll
      for (int u = 0; u < 8; ++u, a += ld) {
        x[u] = __ldcg(a);
        x[8 + u] = __ldcg(a + 32);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u, a += ld) {
        x[u] = (r < M && c + u <= r) ? __ldcg(a) : 0.0;
        x[8 + u] = (r + 32 < M && c + u <= r + 32) ? __ldcg(a + 32) : 0.0;
      }
    }
  }
};

// A grid barrier of all threads.  first() runs in warp 0 between the barrier of
// the CTA and its arrival, over() in the other warps while the barrier is under
// way and in warp 0 after it.
template <class F, class G>
__device__ __forceinline__ bool grid_barrier(GridBarrier* b, unsigned nblocks, unsigned round, int limit_log2, F&& first,
                                             G&& over) {
  __shared__ bool failed;
  __syncthreads();
  if (threadIdx.x >= 32) {
    over();
  } else {
    first();
    __syncwarp();
    if (threadIdx.x == 0) failed = grid_barrier_thread(b, nblocks, round, limit_log2);
  }
  __syncthreads();
  if (threadIdx.x < 32) over();
  return failed;
}

// One panel of NB columns for every problem (cooperative launch).  A CTA owns a
// chunk of rows: it alone reads and writes their rows of V and W, through L1.
// Per column c two phases separated by grid barriers; every load of data written
// by other CTAs during the launch bypasses L1 (__ldcg).
//   A: finish the previous column: y = y' - V p - W q (p = W^T v, q = V^T v
//      of that column), W[:, jj-1] = tau y + a2 v with
//      a2 = -tau^2/2 * (y'^T v - 2 p^T q);  then
//      a = A[c:, c] - V W[c,:]^T - W V[c,:]^T and its norm below c+1.
//   B: Householder vector v of column c (every CTA forms all of it in shared
//      memory), partial p = W^T v, q = V^T v over this CTA's rows, and
//      y' = A22 v with y'^T v from the lower triangle alone, in tiles whose
//      sums go to slots that phase A adds up.  The first tile of a CTA is
//      loaded during the barrier, and strips of it stay in shared memory: A22 is
//      the same for all columns of a panel.
// Deferring the V p + W q correction of y to the next column's phase A saves
// the third grid barrier per column that an eager correction needs.  The
// entries below the subdiagonal of column c are overwritten with v one
// phase later too, because every CTA reads the updated column in phase B.
//
// What bounds a column is the chain of round trips to L2 around the two barriers
// (20000 of 34000 cycles at 2640 rows), then reading A22 and its two sums; while
// the lower triangles together exceed L2, HBM.  Two blocks of 3600 and 3533 rows
// together, down to 1776: 36 us a column when both triangles were read and a
// barrier took seven round trips, 28 with one triangle in tiles that the warps of
// a CTA shared, 17.3 with a tile to a warp, two round trips to a barrier and the
// first strips in shared memory.
// V_SMEM: v in shared memory; otherwise (blocks above 27000 rows) a copy per CTA
// behind the slots of y.
template <bool V_SMEM>
__global__ void __launch_bounds__(TRD_NT, 1) trd_panel_kernel(const TrdProb* __restrict__ probs,
                                                              int nprob, int j0, int nres, int* fail) {
  extern __shared__ double sm[];
  double* scratch = sm;          // 32
  double* VWc = sm + 32;         // 2*NB: row c of V and W
  double* pq = VWc + 2 * NB;     // 2*NB: p, q of the previous column
  double* misc = pq + 2 * NB;    // 8
  double* pqw = misc + 8;        // (TRD_NT/32) x 2*NB partial p, q (phase B)
  double* ypart = pqw;           // 8 x 64 partial sums of y (phase A)
  const int b = blockIdx.x;
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].cta0 <= b) lo = mid; else hi = mid - 1;
  }
  const TrdProb P = probs[lo];
  const int rank = b - P.cta0;
  // Problems are independent: each synchronises only its own CTAs, so a
  // small problem does not wait for a large one inside a panel.
  GridBarrier* bar = P.bar;
  const unsigned nblocks = (unsigned)(P.ncta + P.expect_extra);
  const int n = P.n;
  const size_t ld = (size_t)n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nwarps = TRD_NT / 32, YG = TRD_NT / 64 - 1;
  const int chunk = (n - j0 + P.ncta - 1) / P.ncta;
  const int R0 = min(n, j0 + rank * chunk), R1 = min(n, R0 + chunk);  // this CTA's rows
  const int base = j0 + 1;
  const SymvShape S(max(0, n - base));
  double* yr = P.y;
  double* yc = P.y + (size_t)S.nbn * S.mp;
  double* vs = V_SMEM ? sm + TRD_SMEM : yc + (size_t)S.nbm * S.mp + (size_t)rank * S.mp;  // padded rows
  // this lane's elements of the strips that stay in shared memory
  double* res = sm + TRD_SMEM + (V_SMEM ? S.mp : 0) + warp * nres * 512 + lane;

  // W[:, kp] = tprev (y' - V p - W q) + a2 v of the previous column for this CTA's
  // rows from i0 on, W[i][kp] stored; then f(i, v_i, a) in one lane with
  // a = A[i][c] - V[i] . W[c] - W[i] . V[c].  Warps take four rows at a time.
  // scalars() fills pq, VWc and misc[0] = a2 (the last warp, before the first use).
  auto rows = [&](int i0, int jj, double tprev, auto&& scalars, auto&& f) {
    const int kp = jj - 1;
    for (int rb = R0 + ((i0 - R0) / 64) * 64; rb < R1; rb += 64) {
      // every load of the block at once
      double vik[4], wik[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = rb + warp * 4 + u;
        const bool on = i >= i0 && i < R1;
        vik[u] = on && lane < jj ? P.Vp[(size_t)i * NB + lane] : 0.0;
        wik[u] = on && lane < kp ? P.W[(size_t)i * NB + lane] : 0.0;
      }
      const int il = rb + warp * 4 + lane;  // the row that lanes 0 .. 3 finish
      const bool fin = lane < 4 && il >= i0 && il < R1;
      const double acol = fin && jj < NB ? __ldcg(&P.A[il + (size_t)(j0 + jj) * ld]) : 0.0;
      // the sums by all warps but two, of which one forms the scalars meanwhile
      if (jj > 0 && tid < YG * 64) {
        const int i = rb + (tid & 63), g = tid >> 6;
        ypart[tid] = (i >= i0 && i < R1) ? symv_sum(S, yr, i - base, g, YG) : 0.0;
      }
      if (warp == nwarps - 1 && rb <= i0) scalars();
      __syncthreads();
      const double pk = pq[lane], qk = pq[NB + lane], vck = VWc[lane], wck = VWc[NB + lane];
      const double vckp = jj > 0 ? VWc[kp] : 0.0, a2 = jj > 0 ? misc[0] : 0.0;
      double ys[4], ts[4], vi[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = warp * 4 + u;
        ys[u] = (jj > 0 && lane < YG ? ypart[lane * 64 + rr] : 0.0) - (vik[u] * pk + wik[u] * qk);
        ts[u] = vik[u] * wck + wik[u] * vck;
        vi[u] = jj > 0 ? __shfl_sync(0xffffffffu, vik[u], max(kp, 0)) : 0.0;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          ys[u] += __shfl_xor_sync(0xffffffffu, ys[u], o);
          ts[u] += __shfl_xor_sync(0xffffffffu, ts[u], o);
        }
      if (lane < 4) {
        double y = ys[0], t = ts[0], v = vi[0];
#pragma unroll
        for (int u = 1; u < 4; ++u)
          if (lane == u) {
            y = ys[u];
            t = ts[u];
            v = vi[u];
          }
        if (fin) {
          const double wl = tprev * y + a2 * v;
          if (jj > 0) P.W[(size_t)il * NB + kp] = wl;
          f(il, v, acol - (t + wl * vckp));
        }
      }
      __syncthreads();  // ypart is read
    }
  };

  // A22 and the tiles of a warp stay as they are within a panel: the first nres
  // strips of its first tile are read from global memory for the first column
  // only
  SymvWalk first{P.A + (size_t)base * (ld + 1), ld, S.M, S.nbm, S.nbn, rank + P.ncta * warp, P.ncta * nwarps, 0, 0, 0, {}};
  first.settle();
  for (int jj = 0; jj < NB; ++jj) {
    const int c = j0 + jj;
    const bool act = c < n;
    double* R = P.red + (c & 1) * RED;         // this column's sums
    double* Ro = P.red + ((c + 1) & 1) * RED;  // previous column's sums (next column's slot)
    SymvWalk walk = first;
    if (jj > 0 && first.live()) walk.skip(nres);
    // ---------------- phase A ----------------
    if (act) {
      const int kp = jj - 1;  // columns of V, W before the previous one
      const double tprev = jj > 0 ? __ldcg(&P.tau[c - 1]) : 0.0;
      auto scalars = [&] {
        const double p = (lane < kp) ? ld_volatile(&Ro[2 + lane]) : 0.0, q = (lane < kp) ? ld_volatile(&Ro[2 + NB + lane]) : 0.0;
        const double vc = (lane < jj) ? __ldcg(&P.Vp[(size_t)c * NB + lane]) : 0.0;
        double wc = (lane < kp) ? __ldcg(&P.W[(size_t)c * NB + lane]) : 0.0;
        if (jj > 0) {
          // scalar a2 and row c of the previous column of W (every CTA)
          const double yv = ld_volatile(&Ro[1]), yc = symv_sum(S, yr, c - base, lane, 32);
          const double ptq = warp_sum(p * q);
          const double y = warp_sum(yc - (vc * p + wc * q));
          const double a2 = -0.5 * tprev * tprev * (yv - 2.0 * ptq);
          if (lane == kp) wc = tprev * y + a2 * vc;
          if (lane == 0) misc[0] = a2;
        }
        pq[lane] = p;
        pq[NB + lane] = q;
        VWc[lane] = vc;
        VWc[NB + lane] = wc;
      };
      double ss = 0.0;
      rows(max(R0, c), jj, tprev, scalars, [&](int i, double v, double a) {
        if (jj > 0 && i >= c + 1) P.A[i + (size_t)(c - 1) * ld] = v;
        P.A[i + c * ld] = a;
        if (i == c) P.d[c] = a;
        if (i >= c + 2) ss += a * a;
      });
      ss += __shfl_xor_sync(0xffffffffu, ss, 1);  // of lanes 0 .. 3
      ss += __shfl_xor_sync(0xffffffffu, ss, 2);
      if (lane == 0) scratch[warp] = ss;
    }
    auto add_sum = [&](double* r) {  // of the warps' sums in scratch
      const double x = warp_sum(lane < nwarps ? scratch[lane] : 0.0);
      if (lane == 0 && x != 0.0) atomicAdd(r, x);
    };
    if (grid_barrier(
            bar, nblocks, 2 * jj + 1, P.wait_log2,
            [&] {
              if (act) add_sum(&R[0]);
            },
            [&] {
              if (c < n - 1 && walk.live()) walk.load();
            })) {
      // a wait gave up: end the launch and report it (the host throws)
      if (tid == 0) atomicExch(fail, 1);
      return;
    }
    // ---------------- phase B ----------------
    if (act && c < n - 1) {
      const double alpha = __ldcg(&P.A[c + 1 + c * ld]);
      const double xn2 = ld_volatile(&R[0]);
      double beta = alpha, tc = 0.0, scal = 0.0;
      const bool lost = squares_lost(alpha, xn2);
      if (lost) {  // in every thread of every CTA, with the same sums
        int* tops = reinterpret_cast<int*>(pqw);
        int top = 0;
        for (int r = jj + 1 + tid; r < S.M; r += TRD_NT) top = max(top, upper_word(__ldcg(&P.A[base + r + c * ld])));
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) tops[warp] = top;
        __syncthreads();
        for (int w = 0; w < nwarps; ++w) top = max(top, tops[w]);
        double inverse, ss = 0.0;
        const double p = small_scale(alpha, top, inverse);
        for (int r = jj + 1 + tid; r < S.M; r += TRD_NT) {
          const double x = __ldcg(&P.A[base + r + c * ld]) * p;
          ss += x * x;
        }
        ss = warp_sum(ss);
        if (lane == 0) scratch[warp] = ss;
        __syncthreads();
        reflector_small(alpha, warp_sum(lane < nwarps ? scratch[lane] : 0.0), p, inverse, beta, tc, scal);
      }
      // W and V of this warp's first rows, on the way while v is formed
      double wr[4], vr[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = max(R0, c + 1) + warp + u * nwarps;
        wr[u] = i < R1 && lane < jj ? P.W[(size_t)i * NB + lane] : 0.0;
        vr[u] = i < R1 && lane < jj ? P.Vp[(size_t)i * NB + lane] : 0.0;
      }
      for (int r0 = 0; r0 < S.mp; r0 += 8 * TRD_NT) {
        double a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = r0 + tid + u * TRD_NT;
          a[u] = (r > jj && r < S.M) ? __ldcg(&P.A[base + r + c * ld]) : 0.0;
        }
        if (r0 == 0 && !lost) reflector(alpha, xn2, beta, tc, scal);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = r0 + tid + u * TRD_NT;
          if (r < S.mp) vs[r] = r == jj ? 1.0 : a[u] * scal;
        }
      }
      if (rank == 0 && tid == 0) {
        P.e[c] = beta;
        P.tau[c] = tc;
      }
      if (rank == 0 && tid < RED) Ro[tid] = 0.0;  // read in phase A, refilled from the next phase A on
      __syncthreads();
      double sp = 0.0, sq = 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = max(R0, c + 1) + warp + u * nwarps;
        if (i >= R1) break;
        const double vi = vs[i - base];
        sp += wr[u] * vi;
        sq += vr[u] * vi;
        if (lane == jj) P.Vp[(size_t)i * NB + jj] = vi;
      }
      for (int i = max(R0, c + 1) + warp + 4 * nwarps; i < R1; i += nwarps) {
        const double vi = vs[i - base];
        if (lane < jj) {
          sp += P.W[(size_t)i * NB + lane] * vi;
          sq += P.Vp[(size_t)i * NB + lane] * vi;
        }
        if (lane == jj) P.Vp[(size_t)i * NB + jj] = vi;
      }
      pqw[warp * 2 * NB + lane] = sp;
      pqw[warp * 2 * NB + NB + lane] = sq;
      __syncthreads();
      if (tid < 2 * NB && (tid & (NB - 1)) < jj) {
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < nwarps; ++w) a += pqw[w * 2 * NB + tid];
        if (a != 0.0) atomicAdd(&R[2 + tid], a);
      }
      double yvp = 0.0, a0 = 0.0, a1 = 0.0;
      // one strip; next() may overwrite x and move `at` on
      auto strip = [&](const SymvWalk& at, double (&x)[16], auto&& next) {
        const int I = at.I, J = at.J, r = at.row(), cc = at.col();
        const bool ends = at.strip == SY_N / 8 - 1;
        const double v0 = vs[r], v1 = vs[r + 32];
        double b0 = 0.0, b1 = 0.0, t[8];
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          const double w0 = vs[cc + u], w1 = vs[cc + u + 1];
          a0 += x[u] * w0;
          a1 += x[8 + u] * w0;
          b0 += x[u + 1] * w1;
          b1 += x[9 + u] * w1;
        }
        a0 += b0;
        a1 += b1;
        if (at.below()) {
#pragma unroll
          for (int u = 0; u < 8; ++u) t[u] = x[u] * v0 + x[8 + u] * v1;
        } else {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const double p = x[u] * v0, q = x[8 + u] * v1;
            t[u] = (cc + u == r ? 0.0 : p) + (cc + u == r + 32 ? 0.0 : q);
            yvp -= (cc + u == r ? p * v0 : 0.0) + (cc + u == r + 32 ? q * v1 : 0.0);
          }
        }
        next();
        // column sums over the lanes on the tensor core: product u adds the sums
        // over groups of four lanes of column u to row u of an 8 x 8 accumulator
        double e[2] = {0, 0}, o[2] = {0, 0};
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          dmma(e, (lane >> 2) == u ? 1.0 : 0.0, t[u]);
          dmma(o, (lane >> 2) == u + 1 ? 1.0 : 0.0, t[u + 1]);
        }
        double cs = (e[0] + o[0]) + (e[1] + o[1]);
        cs += __shfl_xor_sync(0xffffffffu, cs, 1);
        cs += __shfl_xor_sync(0xffffffffu, cs, 2);
        if (!(lane & 3)) yc[I * S.mp + cc + (lane >> 2)] = cs;
        if (ends) {
          yr[J * S.mp + r] = a0;
          yr[J * S.mp + r + 32] = a1;
          yvp += 2.0 * (a0 * v0 + a1 * v1);
          a0 = a1 = 0.0;
        }
      };
      if (jj > 0 && first.live()) {
        SymvWalk at = first;
        for (at.strip = 0; at.strip < nres; ++at.strip) {
#pragma unroll
          for (int u = 0; u < 16; ++u) at.x[u] = res[at.strip * 512 + 32 * u];
          strip(at, at.x, [] {});
        }
      }
      while (walk.live())
        strip(walk, walk.x, [&] {
          if (jj == 0 && walk.t == first.t && walk.strip < nres) {
#pragma unroll
            for (int u = 0; u < 16; ++u) res[walk.strip * 512 + 32 * u] = walk.x[u];
          }
          walk.advance();
          if (walk.live()) walk.load();
        });
      yvp = warp_sum(yvp);
      if (lane == 0) scratch[warp] = yvp;
    }
    if (grid_barrier(
            bar, nblocks, 2 * jj + 2, P.wait_log2,
            [&] {
              if (act && c < n - 1) add_sum(&R[1]);
            },
            [] {})) {
      // a wait gave up: end the launch and report it (the host throws)
      if (tid == 0) atomicExch(fail, 1);
      return;
    }
  }
  // finish the panel's last column: W[:, NB-1] for the trailing update and v
  // below its subdiagonal
  const int c = j0 + NB - 1;
  if (c < n - 1) {
    const double* R = P.red + (c & 1) * RED;
    const double tc = __ldcg(&P.tau[c]);
    auto scalars = [&] {
      const double p = (lane < NB - 1) ? ld_volatile(&R[2 + lane]) : 0.0, q = (lane < NB - 1) ? ld_volatile(&R[2 + NB + lane]) : 0.0;
      const double a2 = -0.5 * tc * tc * (ld_volatile(&R[1]) - 2.0 * warp_sum(p * q));
      pq[lane] = p;
      pq[NB + lane] = q;
      VWc[lane] = VWc[NB + lane] = 0.0;
      if (lane == 0) misc[0] = a2;
    };
    rows(max(R0, c + 1), NB, tc, scalars, [&](int i, double v, double) {
      if (i >= c + 2) P.A[i + c * ld] = v;
    });
  }
  // a barrier that gave up is reported to the host (the barriers are reset per launch)
  if (tid == 0 && *reinterpret_cast<volatile int*>(&bar->error)) atomicExch(fail, 1);
}

// --------------------------------------------------------------------------
// The upper triangle from the lower: the panels keep only the lower one, the
// kernels that take the rest of a block read columns of both.
// --------------------------------------------------------------------------
struct MirrorProb {
  double* A;
  int n, ld;
};

constexpr int MIRROR_T = 32;

__global__ void __launch_bounds__(256) mirror_kernel(const MirrorProb* __restrict__ probs) {
  __shared__ double tile[MIRROR_T][MIRROR_T + 1];
  const MirrorProb P = probs[blockIdx.z];
  const int r0 = blockIdx.x * MIRROR_T, c0 = blockIdx.y * MIRROR_T;  // a tile on or below the diagonal
  if (r0 >= P.n || c0 > r0) return;
  const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
  for (int y = y0; y < MIRROR_T; y += 8)
    if (r0 + x < P.n && c0 + y < P.n) tile[y][x] = P.A[r0 + x + (size_t)(c0 + y) * P.ld];
  __syncthreads();
  for (int y = y0; y < MIRROR_T; y += 8) {
    const int r = r0 + y, c = c0 + x;  // of the lower triangle; written at (c, r)
    if (r < P.n && c < r) P.A[c + (size_t)r * P.ld] = tile[x][y];
  }
}

// A kernel's largest dynamic shared memory on the current device only grows:
// solvers on other threads may launch it with more than this call needs, and
// lowering the attribute under them would fail their launches.
cudaError_t raise_smem_attr(const void* func, int bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, int> set;  // (device, kernel) -> bytes set
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(mu);
  int& cur = set[{dev, func}];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

// --------------------------------------------------------------------------
// Zero fill of many device ranges in one launch (one CTA per range of at
// most ZERO_CHUNK doubles).
// --------------------------------------------------------------------------
struct ZeroSeg {
  double* p;
  long long n;
};
constexpr long long ZERO_CHUNK = 32768;

__global__ void zero_kernel(const ZeroSeg* __restrict__ segs) {
  const ZeroSeg z = segs[blockIdx.x];
  for (long long i = threadIdx.x; i < z.n; i += blockDim.x) z.p[i] = 0.0;
}

void zero_add(std::vector<ZeroSeg>& v, double* p, long long n) {
  for (long long o = 0; o < n; o += ZERO_CHUNK) v.push_back(ZeroSeg{p + o, std::min(ZERO_CHUNK, n - o)});
}

// --------------------------------------------------------------------------
// Divide and conquer
// --------------------------------------------------------------------------
struct DcProb {
  int n;
  double* D;      // eigenvalues in progress (n)
  const double* dT;  // tridiagonal diagonal (n)
  const double* e;   // off-diagonal (n-1)
  double* Q;      // n x n (ld n): eigenvectors of T
  double* W1;     // n x n workspace
  double* U;      // n x n workspace
  double* ds;     // n: poles of the secular equation at [lo, lo+k), ascending, scaled by sc
  double* zs;     // n: their weights
  double* val;    // n: the node's new eigenvalues: roots at [lo, lo+k), deflated values after
  int* src;       // n child column of a sorted position
  int* cmap;      // n child column of a compacted position (nondeflated first)
  double* tau;    // n
  int* orig;      // n
  double* zhat;   // n
  int* kcnt;      // n (value at index lo of a node)
  double* rho;    // n (value at index lo; scaled by sc)
  double* sc;     // n (value at index lo): power of two that brings the node's scale near 1
  int* rank;      // n final column of a compacted position
  int* rotp;      // n rotation pairs (compacted positions)
  int* rotj;      // n
  double* rotc;   // n
  double* rots;   // n
  int* nrot;      // n (value at index lo)
};

struct DcNode {
  int prob, lo, mid, hi;
};

// Merge of a node, step 1: z, sorted order, deflation, compaction.  One CTA per
// node.  The values live in shared memory (40 bytes an entry) when the node has
// at most `cap` entries, else in the node's slices of its work arrays in global
// memory.  Deflation by a close pair changes the pair, so the scan is sequential
// in the pairs that deflate; a warp tests 32 pairs at a time and stops at the
// first close one, which makes the scan of a node without close pairs
// parallel (one thread tested them one by one before: 48 us of an n = 301 node).
constexpr int DC_NT = 256;
constexpr int DC_PREP_CAP = 5600;  // largest node staged in shared memory (219 KB)

__host__ __device__ inline size_t dc_prep_smem(int cap) { return (size_t)cap * (3 * sizeof(double) + 4 * sizeof(int)); }

// Exclusive prefix sum of f(j) over 0 <= j < n by the CTA (each thread a run of
// consecutive j); g(j, prefix) for every j; returns the total.
template <class F, class H>
__device__ __forceinline__ int dc_prefix(int n, int* scratch, F&& f, H&& g) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + DC_NT - 1) / DC_NT, j0 = min(n, tid * per), j1 = min(n, j0 + per);
  int c = 0;
  for (int j = j0; j < j1; ++j) c += f(j);
  int inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = inc;
  __syncthreads();
  int base = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < DC_NT / 32; ++w) {
    base += w < warp ? scratch[w] : 0;
    tot += scratch[w];
  }
  int at = base + inc - c;
  for (int j = j0; j < j1; ++j) {
    const int v = f(j);
    g(j, at);
    at += v;
  }
  __syncthreads();
  return tot;
}

__global__ void __launch_bounds__(DC_NT) dc_prep_kernel(const DcProb* __restrict__ probs,
                                                        const DcNode* __restrict__ nodes,
                                                        GemmProb* gprob, GemmSeg* gseg, int cap) {
  extern __shared__ double dcsm[];
  __shared__ double mx[2][DC_NT / 32];
  __shared__ int scratch[DC_NT / 32], s_rot;
  const DcNode N = nodes[blockIdx.x];
  const DcProb P = probs[N.prob];
  const int n = P.n, lo = N.lo, mid = N.mid, hi = N.hi;
  const int n1 = mid - lo, np = hi - lo;
  const size_t ld = (size_t)n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool staged = np <= cap;
  double* dl = staged ? dcsm : P.D + lo;             // the two children's values
  double* wd = staged ? dcsm + cap : P.val + lo;     // sorted d, z
  double* wz = staged ? dcsm + 2 * (size_t)cap : P.tau + lo;
  int* wi = reinterpret_cast<int*>(dcsm + 3 * (size_t)cap);
  int* wf = staged ? wi : P.orig + lo;               // 1: stays in the secular equation
  int* list = staged ? wi + cap : P.rank + lo;       // sorted positions with a z that is not small
  int* src = staged ? wi + 2 * (size_t)cap : P.src + lo;
  int* pos = staged ? wi + 3 * (size_t)cap : P.cmap + lo;  // compacted position of a sorted one
  const double beta = P.e[mid - 1];
  const double rho = 2.0 * fabs(beta);
  const double sgn = beta >= 0.0 ? 1.0 : -1.0;
  const double isq2 = 0.70710678118654752440;
  if (staged)
    for (int i = tid; i < np; i += DC_NT) dl[i] = P.D[lo + i];
  for (int i = tid; i < np; i += DC_NT) src[i] = i;
  __syncthreads();
  // sorted positions by merging the two ascending halves
  double dmax = 0.0, zmax = 0.0;
  for (int i = tid; i < np; i += DC_NT) {
    const double di = dl[i];
    double zi;
    int p;
    if (i < n1) {
      zi = P.Q[(size_t)(mid - 1) + (size_t)(lo + i) * ld] * isq2;
      int a = n1, b = np;  // second-half values less than di
      while (a < b) {
        const int m = (a + b) >> 1;
        if (dl[m] < di) a = m + 1;
        else b = m;
      }
      p = i + (a - n1);
    } else {
      zi = sgn * P.Q[(size_t)mid + (size_t)(lo + i) * ld] * isq2;
      int a = 0, b = n1;
      while (a < b) {
        const int m = (a + b) >> 1;
        if (dl[m] <= di) a = m + 1;
        else b = m;
      }
      p = (i - n1) + a;
    }
    wd[p] = di;
    wz[p] = zi;
    src[p] = i;
    dmax = fmax(dmax, fabs(di));
    zmax = fmax(zmax, fabs(zi));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
  }
  if (lane == 0) {
    mx[0][warp] = dmax;
    mx[1][warp] = zmax;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < DC_NT / 32; ++w) {
    dmax = fmax(dmax, mx[0][w]);
    zmax = fmax(zmax, mx[1][w]);
  }
  const double big = fmax(dmax, rho * zmax), tol = 8.0 * EPS * big, sc = scale_near_one(big);
  // deflation: small z
  const int m = dc_prefix(
      np, scratch, [&](int j) { return rho * fabs(wz[j]) <= tol ? 0 : 1; },
      [&](int j, int at) {
        const int f = rho * fabs(wz[j]) <= tol ? 0 : 1;
        wf[j] = f;
        if (f) list[at] = j;
      });
  // close pairs, in order: |dt c s| <= tol with c = z_j / t, s = -z_p / t,
  // t = |(z_j, z_p)|, tested as |dt z_j z_p| <= tol t^2 (both |z| exceed
  // tol / rho here, so t^2 is normal)
  if (warp == 0) {
    int nr = 0;
    auto close = [&](int p, int j) {
      const double zp = wz[p], zj = wz[j], dt = wd[j] - wd[p];
      return fabs(dt * zj * zp) <= tol * (zj * zj + zp * zp);
    };
    int i = 1;
    while (i < m) {
      const int q = i + lane;
      const unsigned hit = __ballot_sync(0xffffffffu, q < m && close(list[q - 1], list[q]));
      if (!hit) {
        i += 32;
        continue;
      }
      i += __ffs(hit) - 1;
      // from here one pair after another until a pair is not close
      do {
        if (lane == 0) {
          const int p = list[i - 1], j = list[i];
          const double zp = wz[p], zj = wz[j];
          const double t = hypot(zj, zp);
          const double c = zj / t, s = -zp / t;
          const double dp = wd[p], dj = wd[j];
          wz[j] = t;
          wz[p] = 0.0;
          wd[p] = dp * c * c + dj * s * s;
          wd[j] = dp * s * s + dj * c * c;
          wf[p] = 0;
          P.rotp[lo + nr] = p;
          P.rotj[lo + nr] = j;
          P.rotc[lo + nr] = c;
          P.rots[lo + nr] = s;
        }
        __syncwarp();
        ++nr;
        ++i;
      } while (i < m && close(list[i - 1], list[i]));
      ++i;  // the pair (i - 1, i) was tested just now
    }
    if (lane == 0) s_rot = nr;
  }
  __syncthreads();
  const int nr = s_rot;
  // compaction: nondeflated first (in order), then deflated (in order)
  const int k = dc_prefix(
      np, scratch, [&](int j) { return wf[j]; }, [&](int j, int at) { pos[j] = at; });
  for (int j = tid; j < np; j += DC_NT) {
    const int at = wf[j] ? pos[j] : k + (j - pos[j]);
    const int col = min(max(src[j], 0), np - 1);
    if (staged) {
      P.cmap[lo + at] = col;
      if (wf[j]) {
        P.ds[lo + at] = wd[j] * sc;
        P.zs[lo + at] = wz[j];
      } else {
        P.val[lo + at] = wd[j];
      }
    } else {  // the work arrays double as outputs: through others
      P.zhat[lo + at] = wd[j];
      P.ds[lo + at] = wd[j] * sc;
      P.zs[lo + at] = wz[j];
      P.kcnt[lo + at] = col;
    }
  }
  for (int r = tid; r < nr; r += DC_NT) {
    const int p = P.rotp[lo + r], j = P.rotj[lo + r];
    P.rotp[lo + r] = k + (p - pos[p]);
    P.rotj[lo + r] = wf[j] ? pos[j] : k + (j - pos[j]);
  }
  __syncthreads();
  if (!staged) {
    for (int a = tid; a < np; a += DC_NT) {
      P.cmap[lo + a] = P.kcnt[lo + a];
      P.val[lo + a] = P.zhat[lo + a];
    }
    __syncthreads();
  }
  if (tid == 0) {
    P.kcnt[lo] = k;
    P.rho[lo] = rho * sc;
    P.sc[lo] = sc;
    P.nrot[lo] = nr;
    // GEMM descriptor (columns placed by rank): Q[lo:hi, :] = W1[lo:hi, lo:lo+k] * U[lo:lo+k, lo:lo+k]
    GemmProb g = gprob[blockIdx.x];  // tile0/tiles_n preset by the host
    g.C = P.Q + lo + (size_t)lo * ld;
    g.ldc = n;
    g.m = np;
    g.n = k;
    g.beta = 0.0;
    gprob[blockIdx.x] = g;
    GemmSeg s;
    s.A = P.W1 + lo + (size_t)lo * ld;
    s.lda = n;
    s.B = P.U + lo + (size_t)lo * ld;
    s.ldb = n;
    s.k = k;
    s.transA = 0;
    s.transB = 0;
    s.alpha = 1.0;
    gseg[g.seg0] = s;
  }
}

// Step 2: the child eigenvector columns in compacted order, W1[:, a] =
// Q[:, cmap[a]] (a CTA per 128 rows x DC_PCOLS columns), then the deflation
// rotations in order, one thread per row (nothing to do when there are none).
constexpr int DC_PCOLS = 8;

__global__ void dc_gather_kernel(const DcProb* __restrict__ probs, const DcNode* __restrict__ nodes) {
  const DcNode N = nodes[blockIdx.z];
  const DcProb P = probs[N.prob];
  const int lo = N.lo, np = N.hi - N.lo;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int c0 = blockIdx.y * DC_PCOLS;
  if (r >= np || c0 >= np) return;
  const size_t ld = (size_t)P.n;
  const int* map = P.cmap + lo;
  const double* from = P.Q + (size_t)(lo + r) + (size_t)lo * ld;
  double* to = P.W1 + (size_t)(lo + r) + (size_t)lo * ld;
  const int c1 = min(np, c0 + DC_PCOLS);
  for (int c = c0; c < c1; ++c) to[(size_t)c * ld] = from[(size_t)map[c] * ld];
}

__global__ void dc_rotate_kernel(const DcProb* __restrict__ probs, const DcNode* __restrict__ nodes) {
  const DcNode N = nodes[blockIdx.y];
  const DcProb P = probs[N.prob];
  const int lo = N.lo, np = N.hi - N.lo;
  const int nr = P.nrot[lo];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (nr == 0 || r >= np) return;
  const size_t ld = (size_t)P.n;
  double* w1 = P.W1 + (size_t)(lo + r) + (size_t)lo * ld;  // row r, columns lo..hi
  for (int t = 0; t < nr; ++t) {
    const size_t pc = (size_t)P.rotp[lo + t] * ld, jc = (size_t)P.rotj[lo + t] * ld;
    const double c = P.rotc[lo + t], s = P.rots[lo + t];
    const double x = w1[pc], y = w1[jc];
    w1[pc] = c * x + s * y;
    w1[jc] = c * y - s * x;
  }
}

// Step 3: secular equation roots, one warp per root.
__global__ void dc_secular_warp_kernel(const DcProb* __restrict__ probs, const DcNode* __restrict__ nodes,
                                       int* fail) {
  const int j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const DcNode N = nodes[blockIdx.y];
  const DcProb P = probs[N.prob];
  const int lo = N.lo;
  const int k = P.kcnt[lo];
  if (j >= k) return;
  double t;
  int o;
  bool bad;
  secular_root<32>(P.ds + lo, P.zs + lo, k, j, P.rho[lo], lane, true, t, o, bad);
  if (lane == 0) {
    if (bad) atomicExch(fail, 2);
    P.tau[lo + j] = t;
    P.orig[lo + j] = o;
    P.val[lo + j] = (P.ds[lo + o] + t) / P.sc[lo];
  }
}

// Step 4: Loewner z-hat of the nondeflated entries and the final column of
// every entry (its rank among the node's new eigenvalues), one warp per
// entry; writes D.
__global__ void dc_lowner_kernel(const DcProb* __restrict__ probs, const DcNode* __restrict__ nodes) {
  const int i = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const DcNode N = nodes[blockIdx.y];
  const DcProb P = probs[N.prob];
  const int lo = N.lo, np = N.hi - N.lo;
  if (i >= np) return;
  const int k = P.kcnt[lo];
  const double x = P.val[lo + i];
  unsigned r = 0;
  for (int b = lane; b < np; b += 32) {
    const double y = P.val[lo + b];
    r += (y < x) || (y == x && b < i);
  }
  r = __reduce_add_sync(0xffffffffu, r);
  if (lane == 0) {
    P.rank[lo + i] = (int)r;
    P.D[lo + r] = x;
  }
  if (i >= k) return;
  const double* d = P.ds + lo;
  double prod = lowner_product<32>(d, P.orig + lo, P.tau + lo, k, i, lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) prod *= __shfl_xor_sync(0xffffffffu, prod, o);
  prod *= ((d[P.orig[lo + k - 1]] - d[i]) + P.tau[lo + k - 1]) / P.rho[lo];
  if (lane == 0) P.zhat[lo + i] = copysign(sqrt(fmax(prod, 0.0)), P.zs[lo + i]);
}

// Step 5: eigenvectors of the rank-one problem, one warp per column j < k; the
// deflated columns go from W1 to their place in Q.
__global__ void dc_vectors_kernel(const DcProb* __restrict__ probs, const DcNode* __restrict__ nodes) {
  const int j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const DcNode N = nodes[blockIdx.y];
  const DcProb P = probs[N.prob];
  const int lo = N.lo, np = N.hi - N.lo;
  if (j >= np) return;
  const int k = P.kcnt[lo];
  const size_t ld = (size_t)P.n;
  if (j >= k) {
    const double* s = P.W1 + lo + (size_t)(lo + j) * ld;
    double* t = P.Q + lo + (size_t)(lo + P.rank[lo + j]) * ld;
    for (int i = lane; i < np; i += 32) t[i] = s[i];
    return;
  }
  const double* d = P.ds + lo;
  const double dor = d[P.orig[lo + j]];
  const double tj = P.tau[lo + j];
  double* col = P.U + lo + (size_t)(lo + j) * ld;
  double ss = 0.0;
  for (int i = lane; i < k; i += 32) {
    const double u = -P.zhat[lo + i] * rcp_newton((dor - d[i]) + tj);
    col[i] = u;
    ss += u * u;
  }
  ss = warp_sum(ss);
  const double inv = 1.0 / sqrt(ss);
  for (int i = lane; i < k; i += 32) col[i] *= inv;
}

// --------------------------------------------------------------------------
// Back-transformation helpers
// --------------------------------------------------------------------------
struct BtProb {
  int n;
  const double* A;    // reflectors below the subdiagonal
  const double* tau;  // n-1
  double* V;          // n x n (ld n): reflector c in column c, c <= n-2
  double* G;          // nblk blocks of NBB x NBB: V_k^T V_k
  double* T;          // nblk blocks of NBB x NBB: the WY factors
};

// Reflectors of block k (columns j0 = k NBB .. j0 + nb - 1, nb <= NBB).
__host__ __device__ inline int bt_nblk(int n) { return n > 1 ? (n - 2) / NBB + 1 : 0; }

// V[:, c] = (0, .., 0, 1, A[c+2:, c]) for every reflector c of every problem
// (a CTA per column).
__global__ void bt_buildV_kernel(const BtProb* __restrict__ probs) {
  const BtProb P = probs[blockIdx.y];
  const int c = blockIdx.x;
  const int n = P.n;
  if (c > n - 2) return;
  double* col = P.V + (size_t)c * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double v = 0.0;
    if (i == c + 1) v = 1.0;
    else if (i > c + 1) v = P.A[i + (size_t)c * n];
    col[i] = v;
  }
}

// T of the compact WY form of the reflectors j0 .. j0+nb-1 (the dlarft
// recurrence T[0:j, j] = -tau_j T[0:j, 0:j] G[0:j, j], G = V^T V), with G and
// T in shared memory; four threads per row of T share its dot products.
constexpr int BT_T_NT = 4 * NBB;
constexpr size_t BT_T_SMEM = 2 * (size_t)NBB * (NBB + 1) * sizeof(double);

// One CTA per block k (x) of every problem (y).
__global__ void __launch_bounds__(BT_T_NT) bt_T_kernel(const BtProb* __restrict__ probs) {
  const BtProb P = probs[blockIdx.y];
  const int n = P.n;
  const int j0 = blockIdx.x * NBB;
  const int nb = min(NBB, n - 1 - j0);
  if (nb <= 0) return;
  const double* G = P.G + (size_t)blockIdx.x * NBB * NBB;
  double* T = P.T + (size_t)blockIdx.x * NBB * NBB;
  extern __shared__ double btsm[];
  double(*Ts)[NBB + 1] = reinterpret_cast<double(*)[NBB + 1]>(btsm);
  double(*Gs)[NBB + 1] = reinterpret_cast<double(*)[NBB + 1]>(btsm + NBB * (NBB + 1));
  for (int idx = threadIdx.x; idx < NBB * NBB; idx += BT_T_NT) {
    const int r = idx % NBB, c = idx / NBB;
    Ts[r][c] = 0.0;
    Gs[r][c] = G[r + c * NBB];
  }
  __syncthreads();
  const int i = threadIdx.x >> 2, q = threadIdx.x & 3;
  for (int j = 0; j < nb; ++j) {
    double acc = 0.0;
    for (int l = i + q; l < j; l += 4) acc += Ts[i][l] * Gs[l][j];
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    // column j is written here and read only from step j+1 on
    if (q == 0) {
      const double tj = P.tau[j0 + j];
      if (i < j) Ts[i][j] = -tj * acc;
      else if (i == j) Ts[j][j] = tj;
    }
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < NBB * NBB; idx += BT_T_NT) {
    const int r = idx % NBB, c = idx / NBB;
    T[r + c * NBB] = Ts[r][c];
  }
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Host helper that batches GEMM problems and launches them.
// Launch descriptors of several launches gathered on the host and sent to
// the device in one copy (instead of one small copy per launch).
class DescPack {
 public:
  template <class T>
  size_t add(const std::vector<T>& v) {
    const size_t off = (buf_.size() + 255) & ~size_t(255);
    buf_.resize(off + v.size() * sizeof(T));
    if (!v.empty()) memcpy(buf_.data() + off, v.data(), v.size() * sizeof(T));
    return off;
  }
  // device copy (stream-ordered); offsets from add() index into it
  char* upload(DeviceArena& arena, cudaStream_t st) {
    char* dev = static_cast<char*>(arena.alloc(buf_.size() + 256));
    if (!buf_.empty()) NRGB_CUDA(cudaMemcpyAsync(dev, buf_.data(), buf_.size(), cudaMemcpyHostToDevice, st));
    return dev;
  }

 private:
  std::vector<char> buf_;
};

struct GemmBatch {
  std::vector<GemmProb> probs;
  std::vector<GemmSeg> segs;
  int tiles = 0, stiles = 0;
  void add(double* C, int ldc, int m, int n, double beta, const std::vector<GemmSeg>& ss, int ksplit = 1) {
    if (m <= 0 || n <= 0) return;
    GemmProb p{};
    p.ksplit = ksplit;
    p.C = C;
    p.ldc = ldc;
    p.m = m;
    p.n = n;
    p.beta = beta;
    p.seg0 = (int)segs.size();
    p.nseg = (int)ss.size();
    gemm_assign_tiles(p, tiles, stiles);
    segs.insert(segs.end(), ss.begin(), ss.end());
    probs.push_back(p);
  }
  bool empty() const { return probs.empty(); }
};

}  // namespace

// ------------------------------------------------------------------------
// host orchestration
// ------------------------------------------------------------------------

SyevBatched::SyevBatched() {
  NRGB_CUDA(cudaMalloc(&d_err_, 4 * sizeof(int)));
  NRGB_CUDA(cudaMallocHost(&h_err_, 4 * sizeof(int)));
  int dev = 0;
  NRGB_CUDA(cudaGetDevice(&dev));
  NRGB_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
  // NRGB_TRD_PATH=panel keeps every block on the cooperative panel path
  // (comparisons, or a device where cluster launches are unavailable)
  const char* path = getenv("NRGB_TRD_PATH");
  if (!(path && strcmp(path, "panel") == 0)) {
    cl_nmax_ = trdr_init();
    grid_nmax_ = trd_grid_init(&grid_ctas_);
  }
  if (cl_nmax_ <= SMALL_N) cl_nmax_ = 0;
  if (cl_nmax_ == 0) grid_nmax_ = 0;
  // side streams for the launch groups of the cluster kernel (a shape and a
  // cluster size each, up to 21), so that few groups wait behind another
  if (const char* ns = getenv("NRGB_SIDE_STREAMS")) naux_ = std::max(1, std::min(NAUX, atoi(ns)));
  for (int i = 0; i < NAUX; ++i) {
    NRGB_CUDA(cudaStreamCreateWithFlags(&aux_[i], cudaStreamNonBlocking));
    NRGB_CUDA(cudaEventCreateWithFlags(&join_[i], cudaEventDisableTiming));
  }
  NRGB_CUDA(cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming));
  NRGB_CUDA(cudaStreamCreateWithFlags(&small_st_, cudaStreamNonBlocking));
  NRGB_CUDA(cudaEventCreateWithFlags(&small_done_, cudaEventDisableTiming));
}

SyevBatched::~SyevBatched() {
  if (d_err_) cudaFree(d_err_);
  if (h_err_) cudaFreeHost(h_err_);
  for (int i = 0; i < NAUX; ++i) {
    if (aux_[i]) cudaStreamDestroy(aux_[i]);
    if (join_[i]) cudaEventDestroy(join_[i]);
  }
  if (fork_) cudaEventDestroy(fork_);
  if (small_done_) cudaEventDestroy(small_done_);
  if (small_st_) cudaStreamDestroy(small_st_);
}

namespace {
void plan_tree(int prob, int lo, int hi, std::vector<DcNode>& leaves,
               std::vector<std::pair<int, DcNode>>& merges, int& height) {
  if (hi - lo <= LEAF) {
    leaves.push_back(DcNode{prob, lo, lo, hi});
    height = 0;
    return;
  }
  const int mid = lo + (hi - lo) / 2;
  int h1, h2;
  plan_tree(prob, lo, mid, leaves, merges, h1);
  plan_tree(prob, mid, hi, leaves, merges, h2);
  height = std::max(h1, h2) + 1;
  merges.push_back({height, DcNode{prob, lo, mid, hi}});
}
}  // namespace

size_t SyevBatched::workspace_bytes(const std::vector<int>& ns) {
  ArenaPlan pl;
  for (int n : ns) {
    if (n <= SMALL_N) continue;
    const size_t nn = (size_t)n * n;
    pl.add<double>(nn);   // W1
    pl.add<double>(nn);   // U
    pl.add<double>((size_t)n * NB * 2);
    pl.add<double>((size_t)n * 16);
    pl.add<int>((size_t)n * 10);
    pl.add<double>(2 * RED);
    pl.add<double>(trd_grid_exchange(n));
    pl.add<double>((size_t)NBB * NBB * std::max(1, bt_nblk(n)));  // G
    pl.add<double>((size_t)NBB * NBB * std::max(1, bt_nblk(n)));  // T
    pl.add<double>((size_t)NBB * n * 2);                          // X (last pair)
    pl.add<double>((size_t)NBB * n * 2);                          // Y
    pl.add<double>((size_t)NBB * NBB * ((std::max(1, bt_nblk(n)) + 1) / 2));  // G12
  }
  pl.add<double>(64 * 1024);
  int nmx = 0;
  for (int n : ns) nmx = std::max(nmx, n);
  // per-panel launch descriptors
  pl.add<char>((size_t)(nmx / NB + 2) * (ns.size() * (sizeof(TrdProb) + (size_t)(nmx / TRAIL_STRIP + 1) * (2 * sizeof(GemmSeg) + sizeof(GemmProb))) + 2048));
  // zero-fill descriptors: the per-problem buffers once, the split-K
  // outputs of the back-transformation once; cluster descriptors
  size_t zs = 0;
  for (int n : ns)
    zs += 8 + (size_t)n * n / ZERO_CHUNK + trd_grid_exchange(n) / ZERO_CHUNK + 2 * ((size_t)NBB * NBB / ZERO_CHUNK + 1) * bt_nblk(n) +
          (NBB * (size_t)n / ZERO_CHUNK + 2) * (n / NBB + 3);
  pl.add<ZeroSeg>(zs);
  // divide-and-conquer descriptors (one copy): problems, leaves, and per
  // merge node a node, a GEMM problem and a segment; 3 aligned arrays per level
  size_t ndc = 0;
  for (int n : ns) ndc += 2 * (size_t)(n / LEAF + 2);
  pl.add<char>(ns.size() * sizeof(DcProb) + ndc * (sizeof(DcBaseProb) + sizeof(DcNode) + sizeof(GemmProb) + sizeof(GemmSeg) + sizeof(int*)) +
               256 * 4 * 40 + 1024);
  // back-transformation GEMM descriptors (nine products of ten segments per pair of blocks)
  size_t nbt = 0;
  for (int n : ns) nbt += 5 * (size_t)(bt_nblk(n) + 2);
  pl.add<char>(ns.size() * sizeof(BtProb) + nbt * (sizeof(GemmProb) + sizeof(GemmSeg)) +
               256 * 6 * (size_t)(nmx / NBB + 4));
  pl.add<TrdClProb>(2 * ns.size() + 16);
  pl.add<TrdGridProb>(ns.size() + 16);
  pl.add<MirrorProb>(ns.size() + 16);
  pl.add<BtSlabProb>(ns.size() + 16);
  return pl.bytes + (size_t)ns.size() * 4096 + (1 << 20);
}

int SyevBatched::cl_use() const {
  const int lim = schedule_here().cluster_limit.load(std::memory_order_relaxed);
  return (lim > 0 && lim < cl_nmax_) ? lim : cl_nmax_;
}

void SyevBatched::run(const std::vector<SyevDesc>& probs, cudaStream_t st) {
  launches_ = 0;
  NRGB_CUDA(cudaMemsetAsync(d_err_, 0, 4 * sizeof(int), st));
  std::vector<int> small, big;
  for (int i = 0; i < (int)probs.size(); ++i) {
    if (probs[i].n <= 0) continue;
    (probs[i].n <= SMALL_N ? small : big).push_back(i);
  }
  std::vector<int> ns;
  for (int i : big) ns.push_back(probs[i].n);
  // plus descriptor storage
  const size_t need = workspace_bytes(ns) + probs.size() * 512 + (1 << 20);
  if (arena_.capacity() < need) {
    NRGB_CUDA(cudaStreamSynchronize(st));
    arena_.reserve(need + need / 4);
  }
  arena_.reset();

  // ---------------- small problems ----------------
  if (!small.empty()) {
    std::vector<TinyProb> sp;
    for (int i : small) sp.push_back(TinyProb{probs[i].A, probs[i].w, probs[i].Z, probs[i].n});
    TinyProb* d_sp = nullptr;
    if (sp.size() > (size_t)TINY_INLINE) {
      d_sp = arena_.alloc_n<TinyProb>(sp.size());
      NRGB_CUDA(cudaMemcpyAsync(d_sp, sp.data(), sp.size() * sizeof(TinyProb), cudaMemcpyHostToDevice, st));
    }
    // on its own stream, beside the larger blocks; joined before the flags are read
    cudaStream_t sx = big.empty() ? st : small_st_;
    if (sx != st) {
      NRGB_CUDA(cudaEventRecord(fork_, st));
      NRGB_CUDA(cudaStreamWaitEvent(sx, fork_, 0));
    }
    NRGB_CUDA(syev_tiny_launch(sp.data(), d_sp, (int)sp.size(), d_err_ + 2, sx));
    if (sx != st) NRGB_CUDA(cudaEventRecord(small_done_, sx));
    ++launches_;
  }

  if (!big.empty()) {
    const int nbig = (int)big.size();
    int nmax = 0;
    for (int i : big) nmax = std::max(nmax, probs[i].n);
    // per-problem workspaces
    std::vector<TrdProb> tp(nbig);
    std::vector<DcProb> dp(nbig);
    std::vector<BtProb> bt(nbig);
    std::vector<double*> dT(nbig), eT(nbig), tauT(nbig), bt_X(nbig), bt_Y(nbig), bt_G12(nbig), gex(nbig, nullptr);
    std::vector<ZeroSeg> zeros;  // ranges that must start at zero, cleared in one launch
    // The schedule's limit is read once: another thread may change it at any
    // time, and the buffers below must match the paths chosen further down.
    const int clim = cl_use();
    const int glim = clim > 0 ? grid_nmax_ : 0;
    for (int b = 0; b < nbig; ++b) {
      const SyevDesc& S = probs[big[b]];
      const int n = S.n;
      const size_t nn = (size_t)n * n;
      double* W1 = arena_.alloc_n<double>(nn);
      double* U = arena_.alloc_n<double>(nn);
      double* Vp = arena_.alloc_n<double>((size_t)n * NB);
      double* Wp = arena_.alloc_n<double>((size_t)n * NB);
      double* vec = arena_.alloc_n<double>((size_t)n * 16);
      int* ivec = arena_.alloc_n<int>((size_t)n * 10);
      double* red = arena_.alloc_n<double>(2 * RED);
      const int nblk = std::max(1, bt_nblk(n));
      double* G = arena_.alloc_n<double>((size_t)NBB * NBB * nblk);
      double* T = arena_.alloc_n<double>((size_t)NBB * NBB * nblk);
      bt_X[b] = arena_.alloc_n<double>(2 * (size_t)NBB * n);
      bt_Y[b] = arena_.alloc_n<double>(2 * (size_t)NBB * n);
      bt_G12[b] = arena_.alloc_n<double>((size_t)NBB * NBB * ((nblk + 1) / 2));
      dT[b] = vec;
      eT[b] = vec + n;
      tauT[b] = vec + 2 * n;
      TrdProb& t = tp[b];
      t.A = S.A;
      t.d = dT[b];
      t.e = eT[b];
      t.tau = tauT[b];
      t.Vp = Vp;
      t.W = Wp;
      t.y = W1;  // free until divide and conquer
      t.red = red;
      t.n = n;
      DcProb& q = dp[b];
      q.n = n;
      q.D = S.w;
      q.dT = dT[b];
      q.e = eT[b];
      q.Q = S.Z;
      q.W1 = W1;
      q.U = U;
      q.ds = vec + 5 * n;
      q.zs = vec + 6 * n;
      q.val = vec + 7 * n;
      q.tau = vec + 8 * n;
      q.zhat = vec + 9 * n;
      q.rho = vec + 10 * n;
      q.rotc = vec + 11 * n;
      q.rots = vec + 12 * n;
      q.src = ivec;
      q.cmap = ivec + n;
      q.sc = vec + 13 * n;
      q.orig = ivec + 2 * n;
      q.kcnt = ivec + 3 * n;
      q.rank = ivec + 4 * n;
      q.rotp = ivec + 5 * n;
      q.rotj = ivec + 6 * n;
      q.nrot = ivec + 7 * n;
      BtProb& u = bt[b];
      u.n = n;
      u.A = S.A;
      u.tau = tauT[b];
      u.V = W1;  // free once divide and conquer is done
      u.G = G;
      u.T = T;
      if (glim > 0 && n > clim) {
        gex[b] = arena_.alloc_n<double>(trd_grid_exchange(n));
        zero_add(zeros, gex[b], (long long)trd_grid_exchange(n));
      }
      zero_add(zeros, red, 2 * RED);
      zero_add(zeros, tauT[b], n);
      zero_add(zeros, S.Z, (long long)nn);
    }
    if (!zeros.empty()) {
      ZeroSeg* d_z = arena_.alloc_n<ZeroSeg>(zeros.size());
      NRGB_CUDA(cudaMemcpyAsync(d_z, zeros.data(), zeros.size() * sizeof(ZeroSeg), cudaMemcpyHostToDevice, st));
      NRGB_LAUNCH("zero_fill", st, zero_kernel<<<(unsigned)zeros.size(), 256, 0, st>>>(d_z));
      NRGB_CUDA(cudaGetLastError());
      ++launches_;
    }
    // ---------------- 1) tridiagonalisation ----------------
    // Blocks up to the cluster kernel's capacity: one cluster each.  The
    // groups (a shape and a cluster size, trd_regs.cu) are launched largest
    // first and run concurrently on side streams; the panel launches for the
    // larger blocks follow on the main stream.
    std::vector<char> via_cluster(nbig, 0);
    // Launch the cluster tridiagonalisation for `list`, joined into `st`.
    auto launch_clusters = [&](const std::vector<TrdClProb>& list) {
      if (list.empty()) return;
      std::map<std::pair<int, int>, std::vector<TrdClProb>> grp;  // (-shape, -CTAs): largest first
      for (const TrdClProb& t : list) {
        const TrdrGroup g = trdr_group(t.n);
        grp[{-g.shape, -g.cl}].push_back(t);
      }
      std::vector<TrdClProb> all;
      for (const auto& kv : grp) all.insert(all.end(), kv.second.begin(), kv.second.end());
      TrdClProb* dg = arena_.alloc_n<TrdClProb>(all.size());
      NRGB_CUDA(cudaMemcpyAsync(dg, all.data(), all.size() * sizeof(TrdClProb), cudaMemcpyHostToDevice, st));
      NRGB_CUDA(cudaEventRecord(fork_, st));
      int used = 0;
      for (const auto& kv : grp) {
        const TrdrGroup g{-kv.first.first, -kv.first.second};
        cudaStream_t sx = aux_[used % naux_];
        if (used < naux_) NRGB_CUDA(cudaStreamWaitEvent(sx, fork_, 0));
        double fl = 0, by = 0;
        for (const TrdClProb& t : kv.second) {
          fl += 4.0 / 3.0 * (double)t.n * t.n * t.n;
          by += 8.0 * (double)t.n * t.n;  // the block, read from HBM once
        }
        KernelStats::get().add_work("trd_cluster", fl);
        KernelStats::get().add_work("trd_cluster_hbm", by);
        cudaError_t e = cudaSuccess;
        // between 4 ms and a second: a cluster's CTAs run together, its exchange takes microseconds
        const int tries_log2 = std::max(12, std::min(wait_log2_, 20));
        NRGB_LAUNCH("trd_cluster", sx, e = trdr_launch(g, dg, (int)kv.second.size(), tries_log2,
                                                       inject_shortfall_ ? 1 : 0, d_err_ + 3, sx));
        NRGB_CUDA(e);
        dg += kv.second.size();
        ++launches_;
        ++used;
      }
      for (int i = 0; i < std::min(used, naux_); ++i) {
        NRGB_CUDA(cudaEventRecord(join_[i], aux_[i]));
        NRGB_CUDA(cudaStreamWaitEvent(st, join_[i], 0));
      }
    };
    // Larger blocks go to the many-CTA kernel (trd_grid.cu) whole, those
    // beyond its capacity after panel launches for their leading columns.
    std::vector<int> jstop(nbig);
    {
      std::vector<TrdClProb> whole;
      for (int b = 0; b < nbig; ++b) {
        const int n = tp[b].n;
        jstop[b] = n;
        if (clim > 0 && n <= clim) {
          whole.push_back(TrdClProb{tp[b].A, tp[b].d, tp[b].e, tp[b].tau, n, n});
          via_cluster[b] = 1;
        } else if (glim > 0) {
          jstop[b] = n <= glim ? 0 : ((n - glim + NB - 1) / NB) * NB;
        }
      }
      launch_clusters(whole);
    }
    {
      constexpr size_t SMEM_CAP = 227 * 1024 - 64;
      const bool v_smem = ((size_t)TRD_SMEM + SymvShape(nmax).mp) * sizeof(double) <= SMEM_CAP;
      const void* panel = v_smem ? (const void*)trd_panel_kernel<true> : (const void*)trd_panel_kernel<false>;
      NRGB_CUDA(raise_smem_attr(panel, (int)SMEM_CAP));
      const int cap = sms_;  // one CTA per SM: few to synchronise, and v formed once per SM
      // One cooperative launch per panel of NB columns.  All problems advance
      // column by column in lockstep, so a column costs the maximum over
      // problems of (trailing size)^2 / CTAs: the CTAs of each launch are
      // shared among the problems that still have columns left in
      // proportion to (n - j0)^2, and finished problems get none.
      std::vector<int> order(nbig);
      std::iota(order.begin(), order.end(), 0);
      GridBarrier* bars = arena_.alloc_n<GridBarrier>(nbig);
      int jmax = 0;
      for (int b : order)
        if (!via_cluster[b]) jmax = std::max(jmax, jstop[b]);
      for (int j0 = 0; j0 < std::min(nmax, jmax); j0 += NB) {
        std::vector<int> act;
        for (int b : order)
          if (tp[b].n > j0 && !via_cluster[b] && j0 < jstop[b]) act.push_back(b);
        for (size_t s0 = 0; s0 < act.size(); s0 += cap) {
          const size_t s1 = std::min(act.size(), s0 + cap);
          const int cnt = (int)(s1 - s0);
          double wsum = 0.0;
          for (size_t q = s0; q < s1; ++q) wsum += pow((double)(tp[act[q]].n - j0), 2.0);
          const int extra = cap - cnt;
          std::vector<TrdProb> sub;
          int tot = 0;
          NRGB_CUDA(cudaMemsetAsync(bars, 0, sizeof(GridBarrier) * nbig, st));
          for (size_t q = s0; q < s1; ++q) {
            TrdProb t = tp[act[q]];
            t.bar = bars + act[q];
            t.wait_log2 = wait_log2_;
            t.expect_extra = inject_shortfall_ ? 1 : 0;
            const double w = pow((double)(t.n - j0), 2.0) / wsum;
            int nc = 1 + (int)floor(w * extra);
            nc = std::min(nc, std::max(1, (t.n - j0) / (TRD_NT / 32)));
            t.cta0 = tot;
            t.ncta = nc;
            tot += nc;
            sub.push_back(t);
          }
          TrdProb* d_tp = arena_.alloc_n<TrdProb>(sub.size());
          NRGB_CUDA(cudaMemcpyAsync(d_tp, sub.data(), sub.size() * sizeof(TrdProb), cudaMemcpyHostToDevice, st));
          int np_ = cnt;
          int j0_ = j0;
          int* fail = d_err_ + 3;
          int mrows = 0;
          for (const TrdProb& t : sub) mrows = std::max(mrows, t.n - j0 - 1);
          const size_t fixed = ((size_t)TRD_SMEM + (v_smem ? SymvShape(mrows).mp : 0)) * sizeof(double);
          constexpr size_t STRIP_BYTES = (size_t)(TRD_NT / 32) * 512 * sizeof(double);  // of every warp
          int nres = (int)std::min<size_t>(SY_N / 8, (SMEM_CAP - fixed) / STRIP_BYTES);
          const size_t smem = fixed + nres * STRIP_BYTES;
          void* args[] = {(void*)&d_tp, (void*)&np_, (void*)&j0_, (void*)&nres, (void*)&fail};
          {
            // algorithmic bytes: column c reads the lower triangle of its trailing block once
            double wb = 0;
            for (const TrdProb& t : sub)
              for (int c = j0; c < std::min(j0 + NB, t.n - 1); ++c) wb += 4.0 * (double)(t.n - c - 1) * (t.n - c);
            KernelStats::get().add_work("trd_panel", wb);
          }
          NRGB_LAUNCH("trd_panel", st,
                      NRGB_CUDA(cudaLaunchCooperativeKernel(panel, dim3(tot), dim3(TRD_NT),
                                                            args, smem, st)));
          ++launches_;
          // trailing update A22 -= V W^T + W V^T for rows/cols >= j0+NB of the
          // lower triangle, in strips of columns
          GemmBatch gb;
          for (const TrdProb& t : sub) {
            const int n = t.n;
            for (int r0 = j0 + NB; r0 < n; r0 += TRAIL_STRIP) {
              // Vp, W are row-major n x NB: as column-major matrices they are
              // NB x n with ld NB, so op(A) = stored^T and op(B) = stored.
              GemmSeg s1{}, s2{};
              s1.A = t.Vp + (size_t)r0 * NB;
              s1.lda = NB;
              s1.B = t.W + (size_t)r0 * NB;
              s1.ldb = NB;
              s1.k = NB;
              s1.transA = 1;
              s1.transB = 0;
              s1.alpha = -1.0;
              s2 = s1;
              s2.A = t.W + (size_t)r0 * NB;
              s2.B = t.Vp + (size_t)r0 * NB;
              gb.add(t.A + r0 + (size_t)r0 * n, n, n - r0, std::min(TRAIL_STRIP, n - r0), 1.0, {s1, s2});
            }
          }
          if (!gb.empty()) {
            KernelStats::get().add_work("gemm_f64_trailing",
                                        gemm_flops(gb.probs.data(), (int)gb.probs.size(), gb.segs.data()));
            NRGB_CUDA(gemm_grouped_launch_host(gb.probs.data(), (int)gb.probs.size(), gb.segs.data(), (int)gb.segs.size(),
                                               gb.tiles, st, "gemm_f64_trailing", gb.stiles, arena_));
            ++launches_;
          }
        }
      }
    }
    {
      std::vector<MirrorProb> mp;
      int mm = 0;
      for (int b = 0; b < nbig; ++b) {
        const int j = jstop[b], n = tp[b].n;
        if (via_cluster[b] || j == 0 || j >= n) continue;
        mp.push_back(MirrorProb{tp[b].A + j + (size_t)j * n, n - j, n});
        mm = std::max(mm, n - j);
      }
      if (!mp.empty()) {
        MirrorProb* d_mp = arena_.alloc_n<MirrorProb>(mp.size());
        NRGB_CUDA(cudaMemcpyAsync(d_mp, mp.data(), mp.size() * sizeof(MirrorProb), cudaMemcpyHostToDevice, st));
        const unsigned g = (unsigned)((mm + MIRROR_T - 1) / MIRROR_T);
        NRGB_LAUNCH("trd_mirror", st, mirror_kernel<<<dim3(g, g, (unsigned)mp.size()), 256, 0, st>>>(d_mp));
        NRGB_CUDA(cudaGetLastError());
        ++launches_;
      }
    }
    // the blocks A[j:, j:] (j = jstop, fully updated by the last trailing
    // update) on many CTAs each: as many blocks to a cooperative launch as
    // there are CTAs for, largest first, so that blocks of a launch take
    // similar times
    if (glim > 0) {
      std::vector<TrdGridProb> rest;
      for (int b = 0; b < nbig; ++b) {
        const int j = jstop[b], n = tp[b].n;
        if (via_cluster[b] || j >= n) continue;
        rest.push_back(TrdGridProb{tp[b].A + j + (size_t)j * n, tp[b].d + j, tp[b].e + j, tp[b].tau + j, gex[b], n - j, n,
                                   std::min(wait_log2_, 21), inject_shortfall_ ? 1 : 0, 0, 0, 0});
      }
      std::stable_sort(rest.begin(), rest.end(), [](const TrdGridProb& x, const TrdGridProb& y) { return x.n > y.n; });
      std::vector<std::vector<TrdGridProb>> waves;
      std::vector<int> room;
      for (const TrdGridProb& p : rest) {
        const int c = trd_grid_ctas(p.n);
        size_t w = 0;
        while (w < waves.size() && room[w] < c) ++w;
        if (w == waves.size()) {
          waves.emplace_back();
          room.push_back(grid_ctas_);
        }
        waves[w].push_back(p);
        room[w] -= c;
      }
      std::vector<TrdGridProb> all;
      std::vector<int> ctas;
      for (auto& w : waves) {
        ctas.push_back(trd_grid_place(w));
        all.insert(all.end(), w.begin(), w.end());
      }
      TrdGridProb* dg = arena_.alloc_n<TrdGridProb>(all.size());
      if (!all.empty())
        NRGB_CUDA(cudaMemcpyAsync(dg, all.data(), all.size() * sizeof(TrdGridProb), cudaMemcpyHostToDevice, st));
      for (size_t w = 0; w < waves.size(); ++w) {
        double fl = 0;
        for (const TrdGridProb& p : waves[w]) fl += 4.0 / 3.0 * (double)p.n * p.n * p.n;
        KernelStats::get().add_work("trd_grid", fl);
        NRGB_LAUNCH("trd_grid", st, NRGB_CUDA(trd_grid_launch(dg, (int)waves[w].size(), ctas[w], d_err_ + 3, st)));
        dg += waves[w].size();
        ++launches_;
      }
    }
    if (inject_shortfall_) {
      // fault injection (the waits expect a CTA that was never launched):
      // report the timed-out wait here, before any later stage reads the
      // unfinished reduction, and leave no work of this call in flight on any
      // stream
      int f = 0;
      NRGB_CUDA(cudaMemcpyAsync(&f, d_err_ + 3, sizeof(int), cudaMemcpyDeviceToHost, st));
      NRGB_CUDA(cudaStreamSynchronize(st));
      if (small_st_) NRGB_CUDA(cudaStreamSynchronize(small_st_));
      for (int i = 0; i < NAUX; ++i)
        if (aux_[i]) NRGB_CUDA(cudaStreamSynchronize(aux_[i]));
      if (f) throw CudaError("syev: grid barrier timed out");
    }
    // WY factors of the blocks that take the slab back-transformation, beside
    // the divide and conquer
    const int slab_max = bt_slab_nmax();
    std::vector<BtSlabProb> slab;
    std::vector<BtProb> bp;   // the others
    std::vector<int> bp_of;   // their place in `big`
    int slab_nmax = 0, slab_ctas = 0, slab_cols = 8;
    BtSlabProb* d_slab = nullptr;
    {
      std::vector<int> ord;
      long cols = 0;
      for (int b = 0; b < nbig; ++b) {
        if (tp[b].n <= slab_max) {
          ord.push_back(b);
          cols += tp[b].n;
          slab_nmax = std::max(slab_nmax, tp[b].n);
        } else {
          bp.push_back(bt[b]);
          bp_of.push_back(b);
        }
      }
      slab_cols = bt_slab_columns(cols, slab_nmax);
      std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return tp[x].n > tp[y].n; });
      int blocks = 0;
      for (int b : ord) {
        const int n = tp[b].n;
        slab.push_back(BtSlabProb{tp[b].A, tauT[b], bt[b].T, dp[b].Q, n, blocks, slab_ctas});
        blocks += bt_nblk(n);
        slab_ctas += ceil_div(n, slab_cols);
      }
      if (!slab.empty()) {
        d_slab = arena_.alloc_n<BtSlabProb>(slab.size());
        NRGB_CUDA(cudaMemcpyAsync(d_slab, slab.data(), slab.size() * sizeof(BtSlabProb), cudaMemcpyHostToDevice, st));
        NRGB_CUDA(cudaEventRecord(fork_, st));
        NRGB_CUDA(cudaStreamWaitEvent(aux_[0], fork_, 0));
        NRGB_CUDA(bt_wy_launch(d_slab, (int)slab.size(), blocks, aux_[0]));
        NRGB_CUDA(cudaEventRecord(join_[0], aux_[0]));
        ++launches_;
      }
    }
    // ---------------- 2) divide and conquer ----------------
    // Leaves in one launch, then the merges level by level (all problems'
    // nodes of a level together); every level's descriptors go to the
    // device in one copy up front.
    {
      std::vector<DcNode> leaves;
      std::vector<std::pair<int, DcNode>> merges;
      int hmax = 0;
      for (int b = 0; b < nbig; ++b) {
        int h;
        plan_tree(b, 0, dp[b].n, leaves, merges, h);
        hmax = std::max(hmax, h);
      }
      struct Level {
        std::vector<DcNode> nodes;
        GemmBatch gb;
        int maxnp = 0;
        std::vector<const int*> cmaps;  // where the product's columns go: the ranks
        size_t o_nodes = 0, o_gp = 0, o_gs = 0, o_cm = 0;
      };
      std::vector<Level> levels(hmax + 1);
      for (auto& m : merges) levels[m.first].nodes.push_back(m.second);
      DescPack pk;
      const size_t o_dp = pk.add(dp);
      // the subtrees, those beyond half of DC_BASE first (their own launch)
      std::vector<DcBaseProb> base;
      for (const DcNode& L : leaves)
        base.push_back(DcBaseProb{dp[L.prob].dT, dp[L.prob].e, dp[L.prob].D, dp[L.prob].Q, dp[L.prob].n, L.lo, L.hi - L.lo});
      std::stable_sort(base.begin(), base.end(), [](const DcBaseProb& x, const DcBaseProb& y) { return x.s > y.s; });
      int nwide = 0;
      while (nwide < (int)base.size() && base[nwide].s > DC_BASE / 2) ++nwide;
      const size_t o_base = pk.add(base);
      for (int h = 1; h <= hmax; ++h) {
        Level& L = levels[h];
        for (auto& nd : L.nodes) {
          const int np = nd.hi - nd.lo;
          L.maxnp = std::max(L.maxnp, np);
          GemmSeg sg{};
          L.gb.add(nullptr, 0, np, np, 0.0, {sg});  // shapes fixed on device (n = k <= np)
          L.cmaps.push_back(dp[nd.prob].rank + nd.lo);
        }
        // segments too, even though dc_prep fills them in: the copy sizes them
        L.o_nodes = pk.add(L.nodes);
        L.o_gp = pk.add(L.gb.probs);
        L.o_gs = pk.add(L.gb.segs);
        L.o_cm = pk.add(L.cmaps);
      }
      char* dev = pk.upload(arena_, st);
      const DcProb* d_dp = reinterpret_cast<const DcProb*>(dev + o_dp);
      const DcBaseProb* d_base = reinterpret_cast<const DcBaseProb*>(dev + o_base);
      const int nrest = (int)base.size() - nwide;
      const bool both = nwide > 0 && nrest > 0;  // two launches: side by side
      if (both) {
        NRGB_CUDA(cudaEventRecord(fork_, st));
        NRGB_CUDA(cudaStreamWaitEvent(aux_[1], fork_, 0));
      }
      if (nwide > 0) NRGB_CUDA(dc_base_launch(d_base, nwide, base[0].s, d_err_ + 2, st));
      if (nrest > 0) NRGB_CUDA(dc_base_launch(d_base + nwide, nrest, base[nwide].s, d_err_ + 2, both ? aux_[1] : st));
      if (both) {
        NRGB_CUDA(cudaEventRecord(join_[1], aux_[1]));
        NRGB_CUDA(cudaStreamWaitEvent(st, join_[1], 0));
      }
      launches_ += 1 + (both ? 1 : 0);
      NRGB_CUDA(raise_smem_attr((const void*)dc_prep_kernel, (int)dc_prep_smem(DC_PREP_CAP)));
      for (int h = 1; h <= hmax; ++h) {
        Level& L = levels[h];
        if (L.nodes.empty()) continue;
        const int nn = (int)L.nodes.size();
        const int maxnp = L.maxnp;
        const DcNode* d_nodes = reinterpret_cast<const DcNode*>(dev + L.o_nodes);
        GemmProb* d_gp = reinterpret_cast<GemmProb*>(dev + L.o_gp);
        GemmSeg* d_gs = reinterpret_cast<GemmSeg*>(dev + L.o_gs);
        const int cap = maxnp <= DC_PREP_CAP ? maxnp : 0;
        NRGB_LAUNCH("dc_prep", st,
                    dc_prep_kernel<<<nn, DC_NT, dc_prep_smem(cap), st>>>(d_dp, d_nodes, d_gp, d_gs, cap));
        NRGB_CUDA(cudaGetLastError());
        dim3 g1(ceil_div(maxnp, 128), nn);
        dim3 gp(ceil_div(maxnp, 128), ceil_div(maxnp, DC_PCOLS), nn);
        NRGB_LAUNCH("dc_permute", st, dc_gather_kernel<<<gp, 128, 0, st>>>(d_dp, d_nodes));
        NRGB_CUDA(cudaGetLastError());
        NRGB_LAUNCH("dc_permute", st, dc_rotate_kernel<<<g1, 128, 0, st>>>(d_dp, d_nodes));
        NRGB_CUDA(cudaGetLastError());
        dim3 gw(ceil_div(maxnp, 8), nn);
        NRGB_LAUNCH("dc_secular", st, dc_secular_warp_kernel<<<gw, 256, 0, st>>>(d_dp, d_nodes, d_err_ + 2));
        NRGB_CUDA(cudaGetLastError());
        NRGB_LAUNCH("dc_lowner", st, dc_lowner_kernel<<<gw, 256, 0, st>>>(d_dp, d_nodes));
        NRGB_CUDA(cudaGetLastError());
        NRGB_LAUNCH("dc_vectors", st, dc_vectors_kernel<<<gw, 256, 0, st>>>(d_dp, d_nodes));
        NRGB_CUDA(cudaGetLastError());
        NRGB_CUDA(gemm_grouped_launch(d_gp, nn, d_gs, L.gb.tiles, st, "gemm_f64_dc",
                                      gemm_tiles32(L.gb.probs.data(), nn), L.gb.stiles,
                                      reinterpret_cast<const int* const*>(dev + L.o_cm), false));
        launches_ += 7;
      }
      // problems that are a single leaf already have D, Q in place
    }
    // ---------------- 3) back-transformation ----------------
    // Column slabs in one launch (bt_apply.cu) for the blocks they hold.
    if (!slab.empty()) {
      NRGB_CUDA(cudaStreamWaitEvent(st, join_[0], 0));
      NRGB_CUDA(bt_apply_launch(d_slab, (int)slab.size(), slab_cols, slab_ctas, slab_nmax, st));
      ++launches_;
    }
    // The larger ones:
    // Z = H_0 H_1 ... H_{n-2} Z in pairs of blocks of NBB reflectors, last pair
    // first: Z[r0:, :] -= V T (V^T Z[r0:, :]), V = [V_k V_k+1] and
    // T = [T_k, -T_k (V_k^T V_k+1) T_k+1; 0, T_k+1].  V (all reflectors, in W1),
    // every T_k and every T12 are formed up front; then three GEMMs per pair.
    // Split-K outputs X live in their own slots (U, free after divide and
    // conquer, holds those of pairs that end by row n; the last pair uses X),
    // zeroed once.  All descriptors go to the device in one copy.  What bounds
    // them is the FP64 tensor pipe; by single blocks the last product had four
    // steps of 16 to a tile, and the five blocks of 1777 to 3600 rows of one call
    // took 18.1 ms instead of 12.7.
    if (!bp.empty()) {
      const int nbt = (int)bp.size();
      int kmax = 0, pmax = 0, nmaxb = 0;
      for (const BtProb& P : bp) nmaxb = std::max(nmaxb, P.n);
      for (int b = 0; b < nbt; ++b) kmax = std::max(kmax, bt_nblk(bp[b].n));
      pmax = (kmax + 1) / 2;
      constexpr int PB = 2 * NBB;  // reflectors of a pair
      auto xslot = [&](int b, int q) {
        const int n = bp[b].n;
        return (q + 1) * PB <= n ? dp[bp_of[b]].U + (size_t)q * PB * n : bt_X[bp_of[b]];
      };
      auto xsplit = [](int mrows) { return std::max(1, std::min(16, mrows / 256)); };
      auto gsplit = [](int mrows) { return std::max(1, std::min(16, mrows / 256)); };
      auto seg = [](const double* A, int lda, int ta, const double* B, int ldb, int k, double alpha) {
        GemmSeg s{};
        s.A = A;
        s.lda = lda;
        s.transA = ta;
        s.B = B;
        s.ldb = ldb;
        s.k = k;
        s.alpha = alpha;
        return s;
      };
      std::vector<ZeroSeg> bz;
      GemmBatch gg, gm, gt;  // every G_k and V_k^T V_k+1; T_k of that; T12
      constexpr size_t NB2 = (size_t)NBB * NBB;
      for (int b = 0; b < nbt; ++b) {
        const BtProb& P = bp[b];
        const int n = P.n, nblk = bt_nblk(n);
        for (int k = 0; k < nblk; ++k) {
          const int j0 = k * NBB, nb = std::min(NBB, n - 1 - j0), r0 = j0 + 1, mrows = n - r0;
          const double* Vk = P.V + r0 + (size_t)j0 * n;
          const int kg = gsplit(mrows);
          double* Gk = P.G + k * NB2;
          if (kg > 1) zero_add(bz, Gk, (long long)NB2);
          gg.add(Gk, NBB, nb, nb, 0.0, {seg(Vk, n, 1, Vk, n, mrows, 1.0)}, kg);
          if (k & 1) {  // with the block before
            double* G12 = bt_G12[bp_of[b]] + (k / 2) * NB2;
            if (kg > 1) zero_add(bz, G12, (long long)NB2);
            gg.add(G12, NBB, NBB, nb, 0.0, {seg(P.V + r0 + (size_t)(j0 - NBB) * n, n, 1, Vk, n, mrows, 1.0)}, kg);
            // G_k-1 and G_k are free once the T are formed
            gm.add(Gk - NB2, NBB, NBB, nb, 0.0, {seg(P.T + (k - 1) * NB2, NBB, 0, G12, NBB, NBB, 1.0)});
            gt.add(Gk, NBB, NBB, nb, 0.0, {seg(Gk - NB2, NBB, 0, P.T + k * NB2, NBB, nb, -1.0)});
          }
        }
        for (int q = 0; q < (nblk + 1) / 2; ++q)
          if (xsplit(n - q * PB) > 1) zero_add(bz, xslot(b, q), (long long)PB * n);
      }
      // per pair (descending): X = V^T Z, Y = -T X, Z += V Y
      struct Step {
        GemmBatch gx, gy, gz;
      };
      std::vector<Step> steps(pmax);
      for (int q = pmax - 1; q >= 0; --q) {
        Step& S = steps[q];
        for (int b = 0; b < nbt; ++b) {
          const BtProb& P = bp[b];
          const int n = P.n, nblk = bt_nblk(n), k = 2 * q;
          if (k >= nblk) continue;
          // from the row before the first reflector's one on, where V is zero: with
          // an even n the operands are aligned
          const int j0 = q * PB, nb = std::min(PB, n - 1 - j0), r0 = j0, mrows = n - r0;
          const int n1 = std::min(NBB, nb), n2 = nb - n1;
          double* Z = probs[big[bp_of[b]]].Z;
          double *X = xslot(b, q), *Y = bt_Y[bp_of[b]];
          const double* V = P.V + r0 + (size_t)j0 * n;
          const double *T1 = P.T + k * NB2, *T12 = P.G + (k + 1) * NB2;
          S.gx.add(X, PB, nb, n, 0.0, {seg(V, n, 1, Z + r0, n, mrows, 1.0)}, xsplit(mrows));
          if (n2 > 0) {
            S.gy.add(Y, PB, n1, n, 0.0, {seg(T1, NBB, 0, X, PB, n1, -1.0), seg(T12, NBB, 0, X + NBB, PB, n2, -1.0)});
            S.gy.add(Y + NBB, PB, n2, n, 0.0, {seg(T1 + NB2, NBB, 0, X + NBB, PB, n2, -1.0)});
          } else {
            S.gy.add(Y, PB, n1, n, 0.0, {seg(T1, NBB, 0, X, PB, n1, -1.0)});
          }
          S.gz.add(Z + r0, n, mrows, n, 1.0, {seg(V, n, 0, Y, PB, nb, 1.0)});
        }
      }
      // one upload: problems, zero ranges, then the GEMM batches
      DescPack pk;
      const size_t o_bp = pk.add(bp);
      const size_t o_bz = pk.add(bz);
      std::vector<std::pair<size_t, size_t>> og;  // (probs, segs) offsets, batch order below
      auto put = [&](const GemmBatch& g) { og.push_back({pk.add(g.probs), pk.add(g.segs)}); };
      put(gg);
      put(gm);
      put(gt);
      for (int q = pmax - 1; q >= 0; --q) {
        put(steps[q].gx);
        put(steps[q].gy);
        put(steps[q].gz);
      }
      char* dev = pk.upload(arena_, st);
      const BtProb* d_bp = reinterpret_cast<const BtProb*>(dev + o_bp);
      size_t gi = 0;
      auto gemm = [&](const GemmBatch& g) {
        const std::pair<size_t, size_t> o = og[gi++];
        if (g.empty()) return;
        KernelStats::get().add_work("gemm_f64_bt", gemm_flops(g.probs.data(), (int)g.probs.size(), g.segs.data()));
        NRGB_CUDA(gemm_grouped_launch(reinterpret_cast<const GemmProb*>(dev + o.first), (int)g.probs.size(),
                                      reinterpret_cast<const GemmSeg*>(dev + o.second), g.tiles, st, "gemm_f64_bt",
                                      gemm_tiles32(g.probs.data(), (int)g.probs.size()), g.stiles, nullptr,
                                      gemm_scaled(g.segs.data(), (int)g.segs.size())));
        ++launches_;
      };
      if (kmax > 0) {
        NRGB_LAUNCH("bt_buildV", st, bt_buildV_kernel<<<dim3(std::max(1, nmaxb - 1), nbt), 128, 0, st>>>(d_bp));
        NRGB_CUDA(cudaGetLastError());
        ++launches_;
        if (!bz.empty()) {
          NRGB_LAUNCH("zero_fill", st,
                      zero_kernel<<<(unsigned)bz.size(), 256, 0, st>>>(reinterpret_cast<const ZeroSeg*>(dev + o_bz)));
          NRGB_CUDA(cudaGetLastError());
          ++launches_;
        }
        gemm(gg);
        NRGB_CUDA(raise_smem_attr((const void*)bt_T_kernel, (int)BT_T_SMEM));
        NRGB_LAUNCH("bt_T", st, bt_T_kernel<<<dim3(kmax, nbt), BT_T_NT, BT_T_SMEM, st>>>(d_bp));
        NRGB_CUDA(cudaGetLastError());
        ++launches_;
        gemm(gm);
        gemm(gt);
        for (int q = pmax - 1; q >= 0; --q) {
          gemm(steps[q].gx);
          gemm(steps[q].gy);
          gemm(steps[q].gz);
        }
      }
    }
  }
  if (!small.empty() && !big.empty()) NRGB_CUDA(cudaStreamWaitEvent(st, small_done_, 0));
  // error flags
  NRGB_CUDA(cudaMemcpyAsync(h_err_, d_err_, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
  NRGB_CUDA(cudaStreamSynchronize(st));
  if (h_err_[2]) throw CudaError("syev: secular equation iteration did not converge");
  if (h_err_[3]) throw CudaError("syev: grid barrier timed out");
}

}  // namespace nrgb
