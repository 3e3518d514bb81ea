// Unblocked Householder tridiagonalisation of blocks too large for a cluster
// (n up to 1776 on 148 SMs): the recurrence of trd_regs.cu with the columns
// spread over as many SMs as the block needs and the exchange through L2.
//
// What bounds a column is again latency, here of one exchange between all CTAs
// of the block through global memory.  There is no barrier: every entry (S_j
// or R_j of a column) is a 16-byte word of a value and the number of the
// column it belongs to, written and read as one; a thread polls the entries
// of its own rows until they carry the expected number.  The two buffers
// alternate by column parity: a CTA writes column t + 2's entries only after
// it has read all of column t + 1's, which every CTA sends after it has read
// all of column t's (a CTA whose columns are done with sends an entry of its
// own instead, so that nobody overtakes it).
//
// The panel launches that took these blocks before cost 24 us a column (two
// grid barriers and a pass over the trailing matrix in L2).
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "trd_grid.cuh"
#include "trd_regs_dev.cuh"

namespace nrgb {

namespace {

// A value and its tag, moved as one 16-byte word.
__device__ __forceinline__ void st_entry(double* p, double v, unsigned long long tag) {
  asm volatile(
      "{\n.reg .b128 w;\nmov.b128 w, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], w;\n}\n" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}
__device__ __forceinline__ double ld_entry(const double* p, unsigned long long& tag) {
  unsigned long long v;
  asm volatile("{\n.reg .b128 w;\nld.relaxed.gpu.global.b128 w, [%2];\nmov.b128 {%0, %1}, w;\n}\n"
               : "=l"(v), "=l"(tag)
               : "l"(p)
               : "memory");
  return __longlong_as_double(v);
}

// Shared memory of a CTA for a shape, in doubles.
template <class SH>
__host__ __device__ constexpr int grid_smem_doubles(int wr) {
  return 2 * (SH::ROWS + 1) + (SH::ROWS + 2) + (wr + 1) * SH::COLS + 2 * trdr::NW + 2 * 4;
}

template <int KR, int C, int WR>
__device__ __forceinline__ void trd_grid_block(const TrdGridProb& P, int r, double* sm, int* fail) {
  using namespace trdr;
  using SH = Shape<KR, C, WR>;
  static_assert(C <= 16 && C % 2 == 0, "columns of a warp");
  constexpr int WC = SH::WC, ROWS = SH::ROWS, COLS = SH::COLS;
  constexpr int GL = 32 / pow2_up(C);
  constexpr int M = (ROWS + NT - 1) / NT;
  double2* VW = reinterpret_cast<double2*>(sm);  // ROWS + 1: (v, w) of the rows; the last entry stays zero
  double* Rs = sm + 2 * (ROWS + 1);              // [WC][C]: row t + 1 of the columns
  double* Sp = Rs + COLS;                        // [WR][WC][C]: the columns' products
  double* X = Sp + WR * COLS;                    // ROWS + 2
  double* ssp = X + ROWS + 2;                    // NW partial norms
  double* yvp = ssp + NW;                        // NW partial sums of y^T v
  double* scl = yvp + NW;                        // by column parity: y_t, R_t .. : (y_t, alpha)
  __shared__ int s_fail;
  const int n = P.n, NC = P.ncta;
  const size_t ld = (size_t)P.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = warp % WR, wc = warp / WR;

  double a[C][KR];
  int jc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = (c * WC + wc) * NC + r;
    jc[c] = j < n ? j : ROWS;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int i = lane + 32 * (k * WR + wr);
      a[c][k] = (i < n && j < n) ? P.A[i + (size_t)j * ld] : 0.0;
    }
  }
  double v[M], S[M], R[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = tid + NT * m;
    v[m] = 0.0;
    S[m] = 0.0;
    R[m] = i < n ? P.A[i] : 0.0;  // before the first reflector: row 0 of the matrix
  }
  for (int i = tid; i < ROWS + 2; i += NT) X[i] = 0.0;
  for (int i = tid; i <= ROWS; i += NT) VW[i] = make_double2(0.0, 0.0);
  if (tid == 0) s_fail = 0;
  // a reflector is stored one column late: other CTAs may still be reading
  // column 0 of the matrix above, and have done so once its products have come
  __syncthreads();

  double tc = 0.0, scal = 0.0;
  const long long limit = 1ll << P.wait_log2;
  const size_t stride = trd_grid_stride(n);
  auto last_column = [&](int q) { return q + ((n - 1 - q) / NC) * NC; };
  const int jlast = last_column(r), jtok = tid < NC ? last_column(tid) : n;
  int tr = 0;  // t % NC
  for (int t = 0; t < n; ++t) {
    double* sc = scl + 4 * (t & 1);
    // ---- S, R of column t - 1 ----
    if (t > 0) {
      const double* ex = P.ex + ((t - 1) & 1) * stride;
      const unsigned long long want = (unsigned long long)t;
      bool todo[M];
#pragma unroll
      for (int m = 0; m < M; ++m) todo[m] = tid + NT * m >= t && tid + NT * m < n;
      bool tok = jtok < t;  // CTA tid had no live column left in column t - 1
      const bool extra = P.expect_extra && tid == 0;
      long long it = 0;
      while (true) {
        bool wait = false;
#pragma unroll
        for (int m = 0; m < M; ++m)
          if (todo[m]) {
            const double* p = ex + 4 * (tid + NT * m);
            unsigned long long t0, t1;
            S[m] = ld_entry(p, t0);
            R[m] = ld_entry(p + 2, t1);
            todo[m] = t0 != want || t1 != want;
            wait |= todo[m];
          }
        if (tok) {
          unsigned long long t0;
          ld_entry(ex + 4 * (n + 1) + 2 * tid, t0);
          tok = t0 != want;
          wait |= tok;
        }
        if (extra) {
          unsigned long long t0;
          ld_entry(ex + 4 * n, t0);
          wait |= t0 != want;
        }
        if (!wait) break;
        if (++it > limit) {  // a wait that gives up: this CTA ends, the others run out too
          s_fail = 1;
          break;
        }
      }
    }
    double y[M], yv = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = tid + NT * m;
      y[m] = fma(scal, S[m], R[m]);
      yv = (i >= t && i < n) ? fma(y[m], v[m], yv) : yv;
      if (i == t) sc[0] = y[m];
    }
    yv = warp_sum_mma(yv);
    if (lane == 0) yvp[warp] = yv;
    __syncthreads();
    if (s_fail) {
      if (tid == 0) atomicExch(fail, 1);
      return;
    }
    // the reflector of column t - 1 below the subdiagonal
    if (t > 0 && r == (tr == 0 ? NC - 1 : tr - 1)) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = tid + NT * m;
        if (i > t && i < n) P.A[i + (size_t)(t - 1) * ld] = v[m];
      }
    }
    const double a2 = -0.5 * tc * tc * sum8(yvp);
    const double wt = fma(tc, sc[0], a2);
    double x[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = tid + NT * m;
      x[m] = 0.0;
      if (32 * (warp + NW * m) + 31 >= t && i < ROWS) {
        const double w = fma(tc, y[m], a2 * v[m]);
        const double xx = fma(-v[m], wt, R[m]) - w;
        const bool live = i > t && i < n;
        if (i == t && r == 0) P.d[t] = xx;
        if (i == t + 1) sc[1] = xx;
        x[m] = (live && i > t + 1) ? xx : 0.0;
        VW[i] = live ? make_double2(v[m], w) : make_double2(0.0, 0.0);
        X[i] = x[m];
      }
    }
    if (t == n - 1) break;
    __syncthreads();
    // ---- rank-2 update, products of the columns with x ----
    {
      double vj[C], wj[C], acc[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const double2 q = VW[jc[c]];
        vj[c] = q.x;
        wj[c] = q.y;
        acc[c] = 0.0;
      }
      const int k1 = (t + 1) >> 5, l1 = (t + 1) & 31;  // chunks below k1 are done with
      const int kd = k1 - wr;
      const int ks = kd <= 0 ? 0 : (kd + WR - 1) / WR;
      trdr_update_from<0, KR, C, WR>(ks, a, acc, vj, wj, VW + lane + 32 * wr, X + lane + 32 * wr,
                                     ks * WR == kd && lane == l1, Rs + wc * C);
      const double red = columns_sum<C>(acc, lane);
      if (lane % GL == 0 && lane / GL < C) Sp[(wr * WC + wc) * C + lane / GL] = red;
      double ss = 0.0;
#pragma unroll
      for (int m = 0; m < M; ++m) ss = fma(x[m], x[m], ss);
      ss = warp_sum_mma(ss);
      if (lane == 0) ssp[warp] = ss;
    }
    __syncthreads();
    // ---- this CTA's entries ----
    if (tid < COLS) {
      const int at = (tid % WC) * C + tid / WC, j = tid * NC + r;
      if (j > t && j < n) {
        double s = Sp[at];
#pragma unroll
        for (int g = 1; g < WR; ++g) s += Sp[g * COLS + at];
        double* p = P.ex + (t & 1) * stride + 4 * j;
        st_entry(p, s, (unsigned long long)(t + 1));
        st_entry(p + 2, Rs[at], (unsigned long long)(t + 1));
      }
    }
    if (tid == NT - 1 && jlast < t + 1) st_entry(P.ex + (t & 1) * stride + 4 * (n + 1) + 2 * r, 0.0, (unsigned long long)(t + 1));
    // ---- the reflector of column t, while the entries travel ----
    const double nn = sum8(ssp), alpha = sc[1];
    double beta;
    reflector(alpha, nn, beta, tc, scal);
    if (squares_lost(alpha, nn)) {  // in every thread or in none
      int* xtop = reinterpret_cast<int*>(yvp);
      int top = 0;
#pragma unroll
      for (int m = 0; m < M; ++m) top = max(top, upper_word(x[m]));
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0) xtop[warp] = top;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < NW; ++w) top = max(top, xtop[w]);
      double inverse, ss = 0.0;
      const double p = small_scale(alpha, top, inverse);
#pragma unroll
      for (int m = 0; m < M; ++m) ss = fma(x[m] * p, x[m] * p, ss);
      ss = warp_sum_mma(ss);
      if (lane == 0) ssp[warp] = ss;
      __syncthreads();
      reflector_small(alpha, sum8(ssp), p, inverse, beta, tc, scal);
    }
    if (r == 0 && tid == 0) {
      P.e[t] = beta;
      P.tau[t] = tc;
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = tid + NT * m;
      v[m] = i == t + 1 ? 1.0 : x[m] * scal;
    }
    if (++tr == NC) tr = 0;
  }
}

// The shapes, smallest first: <KR, C, WR> holds 32 KR WR rows and C 8/WR
// columns a CTA.
template <class F>
auto with_grid_shape(int s, F&& f) {
  using namespace trdr;
  switch (s) {
    case 0: return f(Shape<6, 12, 4>{});
    case 1: return f(Shape<7, 12, 4>{});
    case 2: return f(Shape<8, 10, 4>{});
    case 3: return f(Shape<10, 8, 4>{});
    case 4: return f(Shape<12, 6, 4>{});
    default: return f(Shape<14, 6, 4>{});
  }
}
constexpr int NGRID = 6;

__global__ void __launch_bounds__(trdr::NT, 1)
    trd_grid_kernel(const TrdGridProb* __restrict__ probs, int nprob, int* fail) {
  extern __shared__ __align__(16) double sm[];
  const int b = blockIdx.x;
  int q = 0;
  while (q + 1 < nprob && probs[q + 1].cta0 <= b) ++q;
  const TrdGridProb P = probs[q];
  const int r = b - P.cta0;
  switch (P.shape) {
    case 0: trd_grid_block<6, 12, 4>(P, r, sm, fail); break;
    case 1: trd_grid_block<7, 12, 4>(P, r, sm, fail); break;
    case 2: trd_grid_block<8, 10, 4>(P, r, sm, fail); break;
    case 3: trd_grid_block<10, 8, 4>(P, r, sm, fail); break;
    case 4: trd_grid_block<12, 6, 4>(P, r, sm, fail); break;
    default: trd_grid_block<14, 6, 4>(P, r, sm, fail); break;
  }
}

int grid_rows(int s) {
  return with_grid_shape(s, [](auto sh) { return decltype(sh)::ROWS; });
}
int grid_cols(int s) {
  return with_grid_shape(s, [](auto sh) { return decltype(sh)::COLS; });
}
int grid_shape(int n) {
  int s = 0;
  while (s + 1 < NGRID && n > grid_rows(s)) ++s;
  return s;
}
size_t grid_smem() {
  int m = 0;
  for (int s = 0; s < NGRID; ++s)
    m = std::max(m, with_grid_shape(s, [](auto sh) { return grid_smem_doubles<decltype(sh)>(4); }));
  return (size_t)m * sizeof(double);
}

}  // namespace

int trd_grid_ctas(int n) {
  const int c = grid_cols(grid_shape(n));
  return (n + c - 1) / c;
}

int trd_grid_init(int* ctas) {
  int dev = 0, coop = 0, sms = 0, per = 0;
  *ctas = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      !coop || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaFuncSetAttribute(trd_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grid_smem()) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, trd_grid_kernel, trdr::NT, grid_smem()) != cudaSuccess || per < 1) {
    cudaGetLastError();
    return 0;
  }
  sms = std::min(sms, TRD_GRID_CTAS);
  *ctas = sms;
  int n = 0;
  for (int s = 0; s < NGRID; ++s) n = std::max(n, std::min(grid_rows(s), grid_cols(s) * sms));
  return n;
}

int trd_grid_place(std::vector<TrdGridProb>& probs) {
  int tot = 0;
  for (TrdGridProb& p : probs) {
    p.shape = grid_shape(p.n);
    p.cta0 = tot;
    p.ncta = trd_grid_ctas(p.n);
    tot += p.ncta;
  }
  return tot;
}

cudaError_t trd_grid_launch(const TrdGridProb* d, int nprob, int ctas, int* fail, cudaStream_t st) {
  void* args[] = {(void*)&d, (void*)&nprob, (void*)&fail};
  return cudaLaunchCooperativeKernel((void*)trd_grid_kernel, dim3(ctas), dim3(trdr::NT), args, grid_smem(), st);
}

}  // namespace nrgb
