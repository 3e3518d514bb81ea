// Unblocked Householder tridiagonalisation of blocks up to n = 640, one block
// per thread-block cluster.
//
// The lower-case names of the recurrence (dsytd2, lower): per column t the
// reflector (beta, tau, v) of column t, y = A v, w = tau y - tau^2/2 (y^T v) v,
// A -= v w^T + w v^T.
//
// What bounds a block is the chain of n dependent columns, not arithmetic
// ((4/3) n^3 flops, a few percent of the FP64 rate) or memory (each block is
// read once).  So the kernel is built to shorten one column:
//  * The matrix stays in registers: warp (wr, wc) of CTA r holds the columns
//    j = (c WC + wc) CL + r in its row chunks of 32 rows, kk = k WR + wr, one
//    row per lane, so that neither the rank-2 update nor the products touch
//    shared memory for matrix entries.  Up to 100 doubles a thread, 256
//    threads, one CTA per SM.
//  * One exchange per column and no cluster barrier: every CTA sends, for its
//    live columns j, S_j = sum_{i >= t+2} A_ij x_i (x: the updated column t,
//    unscaled) and R_j = A_{t+1,j}, and P = p sum_j S_j x_j.  From these every
//    CTA forms y = scale S + R, y^T v = scale^2 P / p + 2 scale S_{t+1} + R_{t+1},
//    w and the next column itself (all CTAs run the same arithmetic on the
//    same values).  p is the power of two that brings the largest |x| near one:
//    without it P is cubic in the matrix's scale, and entries below 1e-105 gave
//    silently wrong eigenvalues, above 1e103 not-a-numbers; with it the square
//    of a column's norm is what limits the range, as everywhere else.  The
//    scale of v is not needed before the products, so the
//    norm's root and divisions run while the messages travel; R is a row
//    of the symmetric matrix, so the owner of column t+1 broadcasts nothing.
//  * The messages are st.async stores that count on the receiver's mbarrier,
//    one warp writing 512 contiguous bytes per target CTA.  Measured per
//    exchange among 16 CTAs: 16-byte stores scattered over the targets 2256
//    cycles, contiguous ones 1831, bulk copies 1608 but with a proxy fence
//    (~200 cycles) and a CTA barrier before them, barrier.cluster with plain
//    remote stores 1651 for the P values alone.
//  * A single-CTA block (n <= 64) has no exchange to hide the root behind: a
//    ninth warp forms the reflector beside the products.
//
// Measured on one B200 (a block alone; before: the shared-memory kernel with
// one cluster barrier per column): n = 64 0.066 ms, n = 128 0.166, n = 256 0.37,
// n = 301 0.44 (before 1.35), n = 464 0.75 (2.3), n = 512 0.82, n = 640 1.6 (3.3).
// The scaling by p and the test for lost squares are 2 to 8 % of that.
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "trd_regs.cuh"
#include "trd_regs_dev.cuh"

namespace nrgb {

namespace {

namespace trdr {

__host__ __device__ constexpr int threads(bool one) { return one ? NT + 32 : NT; }

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// Address of `a` in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ unsigned mapa(unsigned a, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// Store of two doubles into the shared memory of a CTA of the cluster; its
// bytes count on that CTA's mbarrier when they land.
__device__ __forceinline__ void st_async2(unsigned a, double x, double y, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(a),
               "d"(x), "d"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async1(unsigned a, double x, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a), "d"(x),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One try of at most about a microsecond.
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 1000;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.aligned.release;\nbarrier.cluster.wait.aligned.acquire;\n" ::: "memory");
}

// The power of two that brings the largest |x| of a column to [1, 2) (from the
// upper words of the warps' largest; clamped to normal numbers), and its inverse.
__device__ __forceinline__ int column_top(const int* xtop) {
  const int4 a = *reinterpret_cast<const int4*>(xtop), b = *reinterpret_cast<const int4*>(xtop + 4);
  return max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w)));
}
__device__ __forceinline__ double column_scale(const int* xtop, double& inverse) {
  const int e = min(max(column_top(xtop) >> 20, 1), 2045);
  inverse = __hiloint2double(e << 20, 0);
  return __hiloint2double((2046 - e) << 20, 0);
}

// A CTA's message and shared memory.
template <int KR, int C, int WR>
struct ClShape : Shape<KR, C, WR> {
  using Shape<KR, C, WR>::ROWS;
  using Shape<KR, C, WR>::COLS;
  static constexpr int LP = COLS | 1;      // a sender's entries in the exchange buffer (odd: rows in order hit all banks)
  static constexpr size_t smem(int cl) {
    return 16 * ((size_t)(ROWS + 1) + 2 * (size_t)cl * LP) +
           8 * (2 * 16 + (size_t)(WR + 1) * COLS + (ROWS + 2) + 2 * NW + 4) + 64;
  }
};

}  // namespace trdr

template <int KR, int C, int WR, bool ONE>
__global__ void __launch_bounds__(trdr::threads(ONE), 1)
    trd_regs_kernel(const TrdClProb* __restrict__ probs, int CL, int tries, int extra, int* fail) {
  using namespace trdr;
  using SH = ClShape<KR, C, WR>;
  static_assert(C <= 16 && C % 2 == 0, "columns of a warp");
  constexpr int THREADS = threads(ONE);
  constexpr int WC = SH::WC, ROWS = SH::ROWS, COLS = SH::COLS, LP = SH::LP;
  constexpr int GL = 32 / pow2_up(C);           // lanes of a column's group
  constexpr int M = (ROWS + NT - 1) / NT;       // rows of the vectors a thread computes
  extern __shared__ __align__(16) double sm[];
  __shared__ volatile int gave_up;               // a wait of this CTA ran out
  double2* VW = reinterpret_cast<double2*>(sm);  // ROWS + 1: (v, w) of the rows; the last entry stays zero
  double2* SR = VW + ROWS + 1;                   // [2][CL][LP]: (S, R) of every column, by sender
  double* PS = reinterpret_cast<double*>(SR + 2 * CL * LP);  // [2][16]: P, by sender
  double* Rs = PS + 2 * 16;                      // [WC][C]: row t + 1 of the columns
  double* Sp = Rs + COLS;                        // [WR][WC][C]: the columns' products
  double* X = Sp + WR * COLS;                    // ROWS + 2
  double* Pp = X + ROWS + 2;                     // NW
  double* ssp = Pp + NW;                         // NW partial norms
  double* scl = ssp + NW;                        // tau, scale of v, alpha of even and of odd columns
  const unsigned bar = smem_u32(scl + 4);
  int* xtop = reinterpret_cast<int*>(scl + 6);   // NW: by warp, the upper word of its largest |x|
  if (ONE) CL = 1;
  const int r = ONE ? 0 : (int)(blockIdx.x % CL);
  const TrdClProb P = probs[ONE ? blockIdx.x : blockIdx.x / CL];
  const int n = P.n;
  const size_t ld = (size_t)P.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = warp % WR, wc = warp / WR;

  double a[C][KR];
  int jc[C];  // this warp's columns; ROWS (the zero entry of VW and X) beyond the matrix
  int srx[M];  // rows of the vectors held by this thread, i = tid + NT m: their place in SR
  double v[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = tid + NT * m;
    srx[m] = (i < n && warp < NW) ? (i % CL) * LP + i / CL : 0;
    v[m] = 0.0;
  }
  if (warp < NW) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = (c * WC + wc) * CL + r;
      jc[c] = j < n ? j : ROWS;
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        const int i = lane + 32 * (k * WR + wr);
        a[c][k] = (i < n && j < n) ? P.A[i + (size_t)j * ld] : 0.0;
      }
    }
  }
  for (int i = tid; i < 2 * CL * LP; i += THREADS) SR[i] = make_double2(0.0, 0.0);
  for (int i = tid; i < ROWS + 2; i += THREADS) X[i] = 0.0;
  if (tid < 32) PS[tid] = 0.0;
  for (int i = tid; i <= ROWS; i += THREADS) VW[i] = make_double2(0.0, 0.0);
  __syncthreads();
  if (warp < NW) {
#pragma unroll
    for (int m = 0; m < M; ++m)  // before the first reflector: R is row 0 of the matrix
      if (tid + NT * m < n) SR[CL * LP + srx[m]] = make_double2(0.0, P.A[tid + NT * m]);
  }
  int l0 = CL == 1 ? 1 : 0, lr = CL == 1 ? 0 : 1;  // (t + 1) / CL and (t + 1) % CL of the phase t to be sent
  if (!ONE && tid == 0) {
    gave_up = 0;
    mbar_init(bar, 1);
    mbar_init(bar + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect(bar, CL * ((COLS - 1 / CL) * 16 + 8) + extra);
    mbar_expect(bar + 8, CL * ((COLS - 2 / CL) * 16 + 8) + extra);
  }
  __syncthreads();
  if (!ONE) cluster_sync_all();

  double tc = 0.0, scal = 0.0;
  double unp = 1.0;  // 1 / p of the last column
  int tl = 0, tr = 0;  // t / CL, t % CL
  for (int t = 0; t < n; ++t) {
    const int pb = (t + 1) & 1;  // buffer of phase t - 1
    if (!ONE && t > 0) {
      const unsigned bw = bar + 8 * pb, par = ((t - 1) >> 1) & 1;
      int it = 0;
      bool ok = true;
      while (ok && !__all_sync(0xffffffffu, mbar_try(bw, par))) ok = ++it <= tries;
      if (!ok) {  // this CTA ends after its next barrier, the others run out too
        atomicExch(fail, 1);
        gave_up = 1;
      } else if (tid == 0) {  // phase t + 1 (its first column to be sent: (t + 2) / CL)
        const int f = lr + 1 == CL ? l0 + 1 : l0;
        mbar_expect(bw, CL * ((COLS - f) * 16 + 8));
      }
    }
    // ---- vectors: y, w of the last reflector, column t after it ----
    double x[M];
    if (warp < NW) {
      const double2* sr = SR + pb * CL * LP;
      const double2* ps = reinterpret_cast<const double2*>(PS + pb * 16);
      double Ps = ps[0].x;
      if (!ONE) {
        double p0 = ps[0].y, p1 = 0.0;
#pragma unroll
        for (int q = 1; q < 8; ++q)
          if (2 * q < CL) {
            Ps += ps[q].x;
            if (q & 1) p1 += ps[q].y;
            else p0 += ps[q].y;
          }
        Ps += p0 + p1;
      }
      const double2 st = sr[tr * LP + tl];
      const double yt = fma(scal, st.x, st.y);
      const double ytv = fma(scal * unp, scal * Ps, fma(scal, st.x, yt));
      const double a2 = -0.5 * tc * tc * ytv;
      const double wt = fma(tc, yt, a2);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = tid + NT * m;
        x[m] = 0.0;
        if (32 * (warp + NW * m) + 31 >= t && i < ROWS) {
          const double2 q = sr[srx[m]];
          const double w = fma(tc, fma(scal, q.x, q.y), a2 * v[m]);
          const double xx = fma(-v[m], wt, q.y) - w;
          const bool live = i > t && i < n;
          if (i == t && r == 0) P.d[t] = xx;
          if (i == t + 1) scl[2 + (t & 1)] = xx;
          x[m] = (live && i > t + 1) ? xx : 0.0;
          VW[i] = live ? make_double2(v[m], w) : make_double2(0.0, 0.0);
          X[i] = x[m];
        }
      }
      int top = 0;
#pragma unroll
      for (int m = 0; m < M; ++m) top = max(top, upper_word(x[m]));
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0) xtop[warp] = top;
    }
    if (t == n - 1) break;
    __syncthreads();
    const int stop = ONE ? 0 : gave_up;
    if (warp < NW) {
      // ---- matrix: rank-2 update, products of the columns with x ----
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
      const double p = column_scale(xtop, unp);
      double accP = 0.0;
#pragma unroll
      for (int c = 0; c < C; ++c) accP = fma(X[jc[c]] * p, acc[c], accP);
      const double red = columns_sum<C>(acc, lane);
      accP = warp_sum_mma(accP);
      if (lane % GL == 0 && lane / GL < C) Sp[(wr * WC + wc) * C + lane / GL] = red;
      if (lane == 0) Pp[warp] = accP;
      if (!ONE) {
        double ss = 0.0;
#pragma unroll
        for (int m = 0; m < M; ++m) ss = fma(x[m], x[m], ss);
        ss = warp_sum_mma(ss);
        if (lane == 0) ssp[warp] = ss;
      }
    } else {
      // ---- the reflector of column t ----
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int k = 0; k < KR * WR; k += 2) {
        const double u0 = X[lane + 32 * k], u1 = k + 1 < KR * WR ? X[lane + 32 * (k + 1 < KR * WR ? k + 1 : k)] : 0.0;
        s0 = fma(u0, u0, s0);
        s1 = fma(u1, u1, s1);
      }
      const double nn = warp_sum_mma(s0 + s1), alpha = scl[2 + (t & 1)];
      double beta;
      reflector(alpha, nn, beta, tc, scal);
      if (squares_lost(alpha, nn)) {
        double inverse;
        const double p = small_scale(alpha, column_top(xtop), inverse);
        double s = 0.0;
        for (int k = 0; k < KR * WR; ++k) {
          const double u = X[lane + 32 * k] * p;
          s = fma(u, u, s);
        }
        reflector_small(alpha, warp_sum_mma(s), p, inverse, beta, tc, scal);
      }
      if (lane == 0) {
        scl[0] = tc;
        scl[1] = scal;
        P.e[t] = beta;
        P.tau[t] = tc;
      }
    }
    __syncthreads();
    // (nothing is armed or sent after a wait that ran out: the transaction counts
    // would leave their range)
    if (stop) break;
    // ---- S, R of this CTA's columns and P: into the buffer (one CTA), or
    // from every warp to its share of the cluster's CTAs ----
    auto column = [&](int l) {
      const int at = (l % WC) * C + l / WC;
      double s = Sp[at];
#pragma unroll
      for (int g = 1; g < WR; ++g) s += Sp[g * COLS + at];
      return make_double2(s, Rs[at]);
    };
    if (ONE) {
      if (tid < COLS) SR[(t & 1) * LP + tid] = column(tid);
      if (tid == NT) PS[(t & 1) * 16] = sum8(Pp);
      __syncthreads();
    } else if (warp < CL) {
      constexpr int NC = (COLS + 31) / 32;
      double2 q[NC];
#pragma unroll
      for (int h = 0; h < NC; ++h)
        if (lane + 32 * h < COLS) q[h] = column(lane + 32 * h);
      const double ps = sum8(Pp);
      const unsigned dst = smem_u32(SR + ((t & 1) * CL + r) * LP + lane), db = bar + 8 * (t & 1),
                     dp = smem_u32(PS + (t & 1) * 16 + r);
      for (int to = warp; to < CL; to += NW) {
        const unsigned rb = mapa(db, to), ra = mapa(dst, to);
#pragma unroll
        for (int h = 0; h < NC; ++h) {
          const int l = lane + 32 * h;
          if (l >= l0 && l < COLS) st_async2(ra + 512 * h, q[h].x, q[h].y, rb);
        }
        if (lane == 0) st_async1(mapa(dp, to), ps, rb);
      }
    }
    if (ONE) {
      tc = scl[0];
      scal = scl[1];
    } else {  // while the messages travel
      const double nn = sum8(ssp), alpha = scl[2 + (t & 1)];
      double beta;
      reflector(alpha, nn, beta, tc, scal);
      if (squares_lost(alpha, nn)) {  // in every thread or in none
        double inverse, ss = 0.0;
        const double p = small_scale(alpha, column_top(xtop), inverse);
#pragma unroll
        for (int m = 0; m < M; ++m) ss = fma(x[m] * p, x[m] * p, ss);
        ss = warp_sum_mma(ss);
        __syncthreads();
        if (lane == 0) ssp[warp] = ss;
        __syncthreads();
        reflector_small(alpha, sum8(ssp), p, inverse, beta, tc, scal);
      }
      if (r == 0 && tid == 0) {
        P.e[t] = beta;
        P.tau[t] = tc;
      }
    }
    if (warp < NW) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = tid + NT * m;
        v[m] = i == t + 1 ? 1.0 : x[m] * scal;
        if (r == tr && i > t + 1 && i < n) P.A[i + (size_t)t * ld] = v[m];
      }
    }
    if (++tr == CL) {
      tr = 0;
      ++tl;
    }
    if (++lr == CL) {
      lr = 0;
      ++l0;
    }
  }
  if (!ONE) {
    // no CTA leaves while another may still write its shared memory
    __syncthreads();
    cluster_sync_all();
    if (gave_up)  // let copies in flight land before this CTA's memory goes
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
}


// The shapes, smallest first: <KR, C, WR> holds blocks up to 32 KR WR rows on
// ceil(n / (C 8/WR)) CTAs.  Up to 256 rows one warp holds all rows of its 8
// columns (64 columns a CTA); above, two warps share the rows (32 columns a
// CTA), because 64 doubles a thread is what 256 threads hold without spills.
// The last two (40 columns, 90 and 100 doubles, a few spills) take blocks
// beyond 512 rows, which 16 CTAs of 32 columns cannot hold: 2.4 us a column
// against 1.6 at n = 512, but far below a panel column's.  10 columns below 512
// rows use fewer CTAs but are slower in the same proportion (n = 464: 12 CTAs
// 0.87 ms, 15 CTAs 0.73 ms).
template <class F>
auto with_shape(int s, F&& f) {
#define NRGB_TRDR(KR, C, WR, ONE) return f(trdr::ClShape<KR, C, WR>{}, trd_regs_kernel<KR, C, WR, ONE>)
  switch (s) {
    case 0: NRGB_TRDR(2, 8, 1, true);
    case 1: NRGB_TRDR(3, 8, 1, false);
    case 2: NRGB_TRDR(4, 8, 1, false);
    case 3: NRGB_TRDR(5, 8, 1, false);
    case 4: NRGB_TRDR(6, 8, 1, false);
    case 5: NRGB_TRDR(7, 8, 1, false);
    case 6: NRGB_TRDR(8, 8, 1, false);
    case 7: NRGB_TRDR(5, 8, 2, false);
    case 8: NRGB_TRDR(6, 8, 2, false);
    case 9: NRGB_TRDR(7, 8, 2, false);
    case 10: NRGB_TRDR(8, 8, 2, false);
    case 11: NRGB_TRDR(9, 10, 2, false);
    default: NRGB_TRDR(10, 10, 2, false);
  }
#undef NRGB_TRDR
}
constexpr int NSHAPES = 13;
constexpr int CL_MAX = 16;  // non-portable above 8

int shape_rows(int s) {
  return with_shape(s, [](auto sh, auto) { return decltype(sh)::ROWS; });
}
int shape_cluster(int s, int n) {
  return with_shape(s, [n](auto sh, auto) { return (n + decltype(sh)::COLS - 1) / decltype(sh)::COLS; });
}

// Launch configuration of a group (the cluster dimension in `at`).
void group_config(TrdrGroup g, int nprob, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3((unsigned)(nprob * g.cl));
  cfg.blockDim = dim3((unsigned)trdr::threads(g.shape == 0));
  cfg.dynamicSmemBytes = with_shape(g.shape, [&](auto sh, auto) { return decltype(sh)::smem(g.cl); });
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

}  // namespace

TrdrGroup trdr_group(int n) {
  for (int s = 0; s < NSHAPES; ++s)
    if (n <= shape_rows(s)) return TrdrGroup{s, shape_cluster(s, n)};
  return TrdrGroup{-1, 0};
}

int trdr_init() {
  int nmax = 0;
  for (int s = 0; s < NSHAPES; ++s) {
    const int rows = shape_rows(s);
    const TrdrGroup g{s, shape_cluster(s, rows)};
    if (g.cl > CL_MAX) break;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    group_config(g, 1, nullptr, cfg, at);
    const bool usable = with_shape(s, [&](auto, auto kern) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) !=
          cudaSuccess)
        return false;
      if (g.cl > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return false;
      int nc = 0;
      return cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc > 0;
    });
    if (!usable) {
      cudaGetLastError();
      break;
    }
    nmax = rows;
  }
  return nmax;
}

cudaError_t trdr_launch(TrdrGroup g, const TrdClProb* d, int nprob, int wait_log2, int expect_extra, int* fail,
                        cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  group_config(g, nprob, st, cfg, at);
  return with_shape(g.shape, [&](auto, auto kern) {
    return cudaLaunchKernelEx(&cfg, kern, d, g.cl, 1 << wait_log2, 16 * expect_extra, fail);
  });
}

}  // namespace nrgb
