// Divide and conquer of small tridiagonal problems, all levels in one CTA and
// in shared memory, from closed-form 2 x 2 leaves up.
//
// What bounds these levels is latency: as one launch per stage (11 a level, and
// an implicit-QR leaf solver whose rotations are one dependent chain) the
// levels up to 76 rows of an n = 301 block took 0.31 ms, although a level's
// arithmetic is a few microseconds.  Here a level is eight stages between CTA
// barriers; four threads share an entry of the merged problems (their sums meet
// in two shuffles), and the update of the eigenvectors runs on the FP64 tensor
// instruction.  Methods as in the merges of larger nodes (syev.cu): tearing,
// deflation of small z and close d, the secular equation by the two-pole
// iteration, Loewner z-hat.
//
// The deflation rotations act on the rows of the small matrix V (Q V is the
// update), so the children's eigenvectors stay two dense halves: out = [Q1
// V_top; Q2 V_bottom].
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "dc_base.cuh"
#include "dc_secular.cuh"
#include "reflector.cuh"

namespace nrgb {

namespace {

constexpr double EPS = 2.220446049250313e-16;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
constexpr int G = 4;  // threads that share an entry
__device__ __forceinline__ int group_count(int x) {
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Shared memory of a solver for up to CAP rows (G CAP threads).  Leading
// dimensions are 4 mod 16 so that the tensor fragments load without bank
// conflicts.
template <int CAP>
struct DcSm {
  static constexpr int NT = G * CAP;
  static constexpr int LDQ = CAP / 2 + 4;  // columns of the children (at most CAP / 2 rows)
  static constexpr int LDV = CAP + 4;
  static constexpr int QA = CAP * LDQ;
  static constexpr int R2 = CAP * LDV > 2 * CAP * LDQ ? CAP * LDV : 2 * CAP * LDQ;
  double Qa[QA];   // eigenvectors of the nodes of a level, column e at e * LDQ, rows from its node's first
  double R[R2];    // V, and (below the last level) the level's result
  double D[CAP], E[CAP], sd[CAP], sz[CAP], cd[CAP], cz[CAP], tau[CAP], zh[CAP], val[CAP], nD[CAP], rc[CAP], rs[CAP];
  int src[CAP], csrc[CAP], orig[CAP], rank[CAP], rp[CAP], rj[CAP], nd[CAP], nr[CAP], ser[CAP];
};

// Node of entry e at depth d of the halving tree of [0, S).
__device__ __forceinline__ void dc_node(int e, int S, int d, int& lo, int& hi) {
  lo = 0;
  hi = S;
  for (int b = 0; b < d; ++b) {
    const int mid = lo + (hi - lo) / 2;
    if (e < mid) hi = mid;
    else lo = mid;
  }
}
__device__ __forceinline__ void dc_segment(int s, int S, int d, int& lo, int& hi) {
  lo = 0;
  hi = S;
  for (int b = d - 1; b >= 0; --b) {
    const int mid = lo + (hi - lo) / 2;
    if ((s >> b) & 1) lo = mid;
    else hi = mid;
  }
}

// A child column index; entries that are not numbers may leave a sorted
// position unset, whatever it holds must stay inside the node.
__device__ __forceinline__ int dc_column(int c, int np) { return min(max(c, 0), np - 1); }

// The sequential deflation scan of one node (taken when some pair of
// neighbours is close): flags, rotated values, rotations.
template <int CAP>
__device__ void dc_scan(DcSm<CAP>& m, int lo, int hi, double rho, double tol) {
  int nr = 0, prev = -1;
  for (int j = lo; j < hi; ++j) {
    m.nd[j] = 0;
    if (rho * fabs(m.sz[j]) <= tol) continue;
    if (prev >= 0) {
      const double zp = m.sz[prev], zj = m.sz[j], dt = m.sd[j] - m.sd[prev];
      if (fabs(dt * zj * zp) <= tol * (zj * zj + zp * zp)) {
        const double t = hypot(zj, zp);
        const double c = zj / t, s = -zp / t;
        m.sz[j] = t;
        m.sz[prev] = 0.0;
        const double dp = m.sd[prev], dj = m.sd[j];
        m.sd[prev] = dp * c * c + dj * s * s;
        m.sd[j] = dp * s * s + dj * c * c;
        m.rp[lo + nr] = dc_column(m.src[prev], hi - lo);
        m.rj[lo + nr] = dc_column(m.src[j], hi - lo);
        m.rc[lo + nr] = c;
        m.rs[lo + nr] = s;
        ++nr;
      } else {
        m.nd[prev] = 1;
      }
    }
    prev = j;
  }
  if (prev >= 0) m.nd[prev] = 1;
  m.nr[lo] = nr;
}

// Solves the tridiagonal problem in m.D (diagonal, already torn at the ends of
// [0, S)) and m.E.  On return the eigenvalues are in m.D, ascending; the
// eigenvectors go to out (column r at out + r * ldo), shared or global
// memory.  All G CAP threads call it.
template <int CAP>
__device__ void dc_solve(DcSm<CAP>& m, int S, double* out, size_t ldo, int* fail) {
  using SM = DcSm<CAP>;
  constexpr int LDQ = SM::LDQ, LDV = SM::LDV;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e = tid / G, h = tid % G;
  int depth = 0;
  while (((S + (1 << depth) - 1) >> depth) > 2) ++depth;
  // leaves: 1 x 1 and 2 x 2 (symmetric Schur decomposition, Golub & Van Loan 8.4)
  {
    int lo, hi;
    dc_node(min(e, S - 1), S, depth, lo, hi);
    double* q = depth == 0 ? out : m.Qa;
    const size_t lq = depth == 0 ? ldo : (size_t)LDQ;
    double d0 = 0.0, d1 = 0.0;
    const bool mine = e < S && h == 0 && e == lo;
    if (mine) {
      // tearing at the segment's ends inside [0, S)
      d0 = m.D[lo] - (lo > 0 ? fabs(m.E[lo - 1]) : 0.0);
      if (hi - lo == 2) d1 = m.D[lo + 1];
      double& last = hi - lo == 2 ? d1 : d0;
      if (hi < S) last -= fabs(m.E[hi - 1]);
    }
    __syncthreads();
    if (mine) {
      if (hi - lo == 1) {
        m.D[lo] = d0;
        q[lo * lq] = 1.0;
      } else {
        const double b = m.E[lo];
        double cs = 1.0, sn = 0.0, t = 0.0;
        if (b != 0.0) {
          const double th = (d1 - d0) / (2.0 * b);
          t = copysign(1.0, th) / (fabs(th) + sqrt(1.0 + th * th));
          cs = 1.0 / sqrt(1.0 + t * t);
          sn = t * cs;
        }
        const double l0 = d0 - t * b, l1 = d1 + t * b;  // of (cs, -sn) and (sn, cs)
        const bool sw = l1 < l0;
        if (!isfinite(l0) || !isfinite(l1)) atomicExch(fail, 1);
        m.D[lo] = sw ? l1 : l0;
        m.D[lo + 1] = sw ? l0 : l1;
        double* qa = q + (lo + (sw ? 1 : 0)) * lq;
        double* qb = q + (lo + (sw ? 0 : 1)) * lq;
        qa[0] = cs;
        qa[1] = -sn;
        qb[0] = sn;
        qb[1] = cs;
      }
    }
    __syncthreads();
  }
  for (int d = depth - 1; d >= 0; --d) {
    const bool last = d == 0;
    const int npm = (S + (1 << d) - 1) >> d;  // largest node of the level
    const int ldv = npm <= CAP / 2 ? LDQ : LDV;
    double* V = m.R;
    int lo, hi;
    dc_node(min(e, S - 1), S, d, lo, hi);
    const int mid = lo + (hi - lo) / 2;
    const bool on = e < S;
    const double beta = m.E[mid - 1];
    const double rho = 2.0 * fabs(beta);
    // 1. z, sorted order of the two ascending halves
    if (on && h == 0) {
      const double di = m.D[e];
      double zi;
      int pos;
      if (e < mid) {
        zi = m.Qa[e * LDQ + (mid - 1 - lo)];
        int a = mid, b = hi;
        while (a < b) {
          const int q = (a + b) >> 1;
          if (m.D[q] < di) a = q + 1;
          else b = q;
        }
        pos = (e - lo) + (a - mid);
      } else {
        zi = copysign(1.0, beta) * m.Qa[e * LDQ];
        int a = lo, b = mid;
        while (a < b) {
          const int q = (a + b) >> 1;
          if (m.D[q] <= di) a = q + 1;
          else b = q;
        }
        pos = (e - mid) + (a - lo);
      }
      m.sd[lo + pos] = di;
      m.sz[lo + pos] = zi * 0.70710678118654752440;
      m.src[lo + pos] = e - lo;
      m.ser[e] = 0;
      m.nr[e] = 0;
    }
    for (int i = tid; i < S * ldv; i += SM::NT) V[i] = 0.0;
    __syncthreads();
    // 2. deflation
    double tol, sc;  // deflation threshold, scale of the secular problem
    {
      double zm = 0.0;
      for (int q = lo + h; q < hi; q += G) zm = fmax(zm, fabs(m.sz[q]));
#pragma unroll
      for (int o = G / 2; o >= 1; o >>= 1) zm = fmax(zm, __shfl_xor_sync(0xffffffffu, zm, o));
      const double dm = fmax(fmax(fabs(m.D[lo]), fabs(m.D[mid - 1])), fmax(fabs(m.D[mid]), fabs(m.D[hi - 1])));
      tol = 8.0 * EPS * fmax(dm, rho * zm);
      sc = scale_near_one(fmax(dm, rho * zm));
    }
    if (on && h == 0) {
      const bool keep = !(rho * fabs(m.sz[e]) <= tol);
      m.nd[e] = keep;
      if (keep) {
        int p = e - 1;
        while (p >= lo && rho * fabs(m.sz[p]) <= tol) --p;
        if (p >= lo) {
          const double zp = m.sz[p], zj = m.sz[e], dt = m.sd[e] - m.sd[p];
          if (fabs(dt * zj * zp) <= tol * (zj * zj + zp * zp)) m.ser[lo] = 1;
        }
      }
    }
    __syncthreads();
    if (on && h == 0 && e == lo && m.ser[lo]) dc_scan(m, lo, hi, rho, tol);
    __syncthreads();
    // 3. compaction: the nondeflated first, then the deflated, both in order
    int k;
    {
      int tot = 0, before = 0;
      for (int q = lo + h; q < hi; q += G) {
        const int f = m.nd[q];
        tot += f;
        before += q < e ? f : 0;
      }
      k = group_count(tot);
      before = group_count(before);
      if (on && h == 0) {
        const int a = m.nd[e] ? before : k + (e - lo - before);
        m.csrc[lo + a] = dc_column(m.src[e], hi - lo);
        if (a < k) {
          m.cd[lo + a] = m.sd[e] * sc;
          m.cz[lo + a] = m.sz[e];
        } else {
          m.val[lo + a] = m.sd[e];
        }
      }
    }
    __syncthreads();
    // 4. roots
    const int a = e - lo;
    const bool root = on && a < k;
    double ta;
    int oa;
    bool bad;
    secular_root<G>(m.cd + lo, m.cz + lo, k, a, rho * sc, h, root, ta, oa, bad);
    if (root && h == 0) {
      if (bad) atomicExch(fail, 1);
      m.tau[e] = ta;
      m.orig[e] = oa;
      m.val[e] = (m.cd[lo + oa] + ta) / sc;
    }
    __syncthreads();
    // 5. Loewner z-hat; final order
    {
      const double* cd = m.cd + lo;
      double prod = root ? lowner_product<G>(cd, m.orig + lo, m.tau + lo, k, a, h) : 1.0;
#pragma unroll
      for (int o = G / 2; o >= 1; o >>= 1) prod *= __shfl_xor_sync(0xffffffffu, prod, o);
      if (root && h == 0) {
        prod *= ((cd[m.orig[lo + k - 1]] - cd[a]) + m.tau[lo + k - 1]) / (rho * sc);
        m.zh[e] = copysign(sqrt(fmax(prod, 0.0)), m.cz[e]);
      }
      const double x = on ? m.val[e] : 0.0;
      int r = 0;
      for (int q = lo + h; q < hi; q += G) {
        const double y = m.val[q];
        r += (y < x) || (y == x && q < e);
      }
      r = group_count(r);
      if (on && h == 0) {
        m.rank[e] = lo + r;
        m.nD[lo + r] = x;
      }
    }
    __syncthreads();
    // 6. V: eigenvectors of the rank-one problem by child column, unit columns for the deflated
    {
      double ss = 0.0;
      if (root) {
        const double dor = m.cd[lo + oa];
        for (int i = h; i < k; i += G) {
          const double u = -m.zh[lo + i] * rcp_newton((dor - m.cd[lo + i]) + ta);
          V[e * ldv + m.csrc[lo + i]] = u;
          ss += u * u;
        }
      }
      ss = group_sum<G>(ss);
      if (root) {
        const double inv = 1.0 / sqrt(ss);
        for (int i = h; i < k; i += G) V[e * ldv + m.csrc[lo + i]] *= inv;
      } else if (on && h == 0) {
        V[e * ldv + m.csrc[lo + a]] = 1.0;
      }
      __syncwarp();
      if (on && h == 0)
        for (int r = m.nr[lo] - 1; r >= 0; --r) {
          double* vp = V + e * ldv + m.rp[lo + r];
          double* vj = V + e * ldv + m.rj[lo + r];
          const double c = m.rc[lo + r], s = m.rs[lo + r], x = *vp, y = *vj;
          *vp = c * x - s * y;
          *vj = s * x + c * y;
        }
    }
    __syncthreads();
    // 7. out = [Q1 V_top; Q2 V_bottom], columns in final order
    {
      double* to = last ? out : m.R + CAP * LDQ;
      const size_t ldt = last ? ldo : (size_t)LDQ;
      if (npm <= 16) {
        // few terms: each entry's threads form their column
        if (on)
          for (int row = h; row < hi - lo; row += G) {
            const bool top = row < mid - lo;
            const double* qp = m.Qa + (top ? lo : mid) * LDQ + (top ? row : row - (mid - lo));
            const double* vp = V + e * ldv + (top ? 0 : mid - lo);
            const int cnt = top ? mid - lo : hi - mid;
            double s = 0.0;
            for (int i = 0; i < cnt; ++i) s = fma(qp[i * LDQ], vp[i], s);
            to[m.rank[e] * ldt + row] = s;
          }
      } else {
        // a warp takes 16 columns of a node, all its row tiles; rows and
        // columns outside the node read clamped addresses and are not stored
        const int nodes = 1 << d, nt2 = (npm + 15) / 16, g = lane >> 2, t = lane & 3;
        for (int p = warp; p < nodes * nt2; p += SM::NT / 32) {
          const int s = p / nt2;
          int nlo, nhi;
          dc_segment(s, S, d, nlo, nhi);
          const int nmid = nlo + (nhi - nlo) / 2, col = nlo + 16 * (p - s * nt2);
          if (col >= nhi) continue;
          for (int half = 0; half < 2; ++half) {
            const int c0 = half ? nmid : nlo, rows = half ? nhi - nmid : nmid - nlo;  // child columns, rows
            const double* vp = V + min(col + g, nhi - 1) * ldv + (c0 - nlo) + t;
            const double* vq = V + min(col + 8 + g, nhi - 1) * ldv + (c0 - nlo) + t;
            for (int m0 = 0; m0 < rows; m0 += 8) {
              const int row = m0 + g;
              const double* qp = m.Qa + (c0 + t) * LDQ + min(row, rows - 1);
              double acc[2][4] = {};
              int q = 0;
              for (; q + 8 <= rows; q += 8) {
                const double a0 = qp[q * LDQ], a1 = qp[(q + 4) * LDQ];
                dmma(acc[0][0], acc[0][1], a0, vp[q]);
                dmma(acc[0][2], acc[0][3], a0, vq[q]);
                dmma(acc[1][0], acc[1][1], a1, vp[q + 4]);
                dmma(acc[1][2], acc[1][3], a1, vq[q + 4]);
              }
              for (; q < rows; q += 4) {
                const bool in = q + t < rows;
                const double a0 = in ? qp[q * LDQ] : 0.0, b0 = in ? vp[q] : 0.0, b1 = in ? vq[q] : 0.0;
                dmma(acc[0][0], acc[0][1], a0, b0);
                dmma(acc[0][2], acc[0][3], a0, b1);
              }
              if (row < rows) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const int cc = col + 8 * (u >> 1) + 2 * t + (u & 1);
                  if (cc < nhi) to[m.rank[cc] * ldt + (c0 - nlo) + row] = acc[0][u] + acc[1][u];
                }
              }
            }
          }
        }
      }
    }
    __syncthreads();
    if (on && h == 0) m.D[e] = m.nD[e];
    if (!last)
      for (int i = tid; i < S * LDQ; i += SM::NT) m.Qa[i] = m.R[CAP * LDQ + i];
    __syncthreads();
  }
}

template <int CAP>
__global__ void __launch_bounds__(G * CAP) dc_base_kernel(const DcBaseProb* __restrict__ probs, int* fail) {
  extern __shared__ __align__(16) unsigned char raw[];
  DcSm<CAP>& m = *reinterpret_cast<DcSm<CAP>*>(raw);
  const DcBaseProb P = probs[blockIdx.x];
  const int i = threadIdx.x;
  if (i < P.s) {
    double d = P.d[P.lo + i];
    if (i == 0 && P.lo > 0) d -= fabs(P.e[P.lo - 1]);
    if (i == P.s - 1 && P.lo + P.s < P.n) d -= fabs(P.e[P.lo + P.s - 1]);
    m.D[i] = d;
    m.E[i] = i < P.s - 1 ? P.e[P.lo + i] : 0.0;
  }
  __syncthreads();
  dc_solve<CAP>(m, P.s, P.Q + P.lo + (size_t)P.lo * P.n, (size_t)P.n, fail);
  if (i < P.s) P.D[P.lo + i] = m.D[i];
}

// Householder tridiagonalisation of a block of up to N rows by warp 0, one row
// a lane in registers; divide and conquer by the CTA (4 N threads); the reflectors
// applied to the eigenvectors, a column a thread.
template <int N>
struct TinySm {
  DcSm<N> dc;
  double Z[N * (N + 1)];
  double v[N][N + 2];  // reflectors
  double w[N], tau[N];
};

template <int N>
__device__ __forceinline__ void syev_tiny(const TinyProb P, int* fail) {
  extern __shared__ __align__(16) unsigned char raw[];
  TinySm<N>& m = *reinterpret_cast<TinySm<N>*>(raw);
  const int n = P.n, tid = threadIdx.x, lane = tid & 31;
  if (tid < 32) {
    double a[N];
#pragma unroll
    for (int j = 0; j < N; ++j) a[j] = (lane < n && j < n) ? P.A[lane + (size_t)j * n] : 0.0;
    double ac = a[0];  // column c, rows by lane
    for (int c = 0; c < n; ++c) {
      if (lane == c) m.dc.D[c] = ac;
      if (c == n - 1) break;
      const double xi = lane >= c + 2 ? ac : 0.0;
      const double xn2 = warp_sum(xi * xi);
      const double alpha = __shfl_sync(0xffffffffu, ac, c + 1);
      double tc, beta, scal;
      reflector(alpha, xn2, beta, tc, scal);
      if (squares_lost(alpha, xn2)) {
        double inverse;
        const double p = small_scale(alpha, (int)__reduce_max_sync(0xffffffffu, upper_word(xi)), inverse);
        reflector_small(alpha, warp_sum(xi * p * (xi * p)), p, inverse, beta, tc, scal);
      }
      const double vi = lane == c + 1 ? 1.0 : xi * scal;
      if (lane < N) m.v[c][lane] = vi;
      if (lane == 0) {
        m.dc.E[c] = beta;
        m.tau[c] = tc;
      }
      __syncwarp();
      // p = tau A v; w = p - tau/2 (p^T v) v
      double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
#pragma unroll
      for (int j = 0; j < N; j += 4) {
        const double2 x = *reinterpret_cast<const double2*>(&m.v[c][j]);
        const double2 y = *reinterpret_cast<const double2*>(&m.v[c][j + 2]);
        p0 = fma(a[j], x.x, p0);
        p1 = fma(a[j + 1], x.y, p1);
        p2 = fma(a[j + 2], y.x, p2);
        p3 = fma(a[j + 3], y.y, p3);
      }
      const double pi = lane > c ? tc * ((p0 + p1) + (p2 + p3)) : 0.0;
      const double wi = pi - 0.5 * tc * warp_sum(pi * vi) * vi;
      if (lane < N) m.w[lane] = wi;
      __syncwarp();
      double nx = 0.0;
#pragma unroll
      for (int j = 0; j < N; j += 2) {
        const double2 x = *reinterpret_cast<const double2*>(&m.v[c][j]);
        const double2 y = *reinterpret_cast<const double2*>(&m.w[j]);
        a[j] = fma(-vi, y.x, fma(-wi, x.x, a[j]));
        a[j + 1] = fma(-vi, y.y, fma(-wi, x.y, a[j + 1]));
        if (j == c + 1) nx = a[j];
        if (j + 1 == c + 1) nx = a[j + 1];
      }
      ac = nx;
      __syncwarp();
    }
    if (lane == 0) m.dc.E[n - 1] = 0.0;
  }
  __syncthreads();
  dc_solve<N>(m.dc, n, m.Z, N + 1, fail);
  if (tid < n) {
    P.w[tid] = m.dc.D[tid];
    double z[N];
#pragma unroll
    for (int i = 0; i < N; ++i) z[i] = i < n ? m.Z[tid * (N + 1) + i] : 0.0;
    for (int c = n - 2; c >= 0; --c) {
      const double tc = m.tau[c];
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const double2 x = *reinterpret_cast<const double2*>(&m.v[c][i]);
        s0 = fma(x.x, z[i], s0);
        s1 = fma(x.y, z[i + 1], s1);
      }
      const double s = -tc * (s0 + s1);
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const double2 x = *reinterpret_cast<const double2*>(&m.v[c][i]);
        z[i] = fma(s, x.x, z[i]);
        z[i + 1] = fma(s, x.y, z[i + 1]);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < n) m.Z[tid * (N + 1) + i] = z[i];
  }
  __syncthreads();
  for (int i = tid; i < n * n; i += G * N) P.Z[i] = m.Z[(i / n) * (N + 1) + i % n];
}

}  // namespace

cudaError_t dc_base_launch(const DcBaseProb* d, int nprob, int smax, int* fail, cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  // two sizes: subtrees up to 64 rows leave room for three CTAs an SM
  const bool half = smax <= DC_BASE / 2;
  const size_t smem = half ? sizeof(DcSm<DC_BASE / 2>) : sizeof(DcSm<DC_BASE>);
  cudaError_t e = half ? cudaFuncSetAttribute(dc_base_kernel<DC_BASE / 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                       : cudaFuncSetAttribute(dc_base_kernel<DC_BASE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (half) NRGB_LAUNCH("dc_leaf", st, dc_base_kernel<DC_BASE / 2><<<nprob, G * DC_BASE / 2, smem, st>>>(d, fail));
  else NRGB_LAUNCH("dc_leaf", st, dc_base_kernel<DC_BASE><<<nprob, G * DC_BASE, smem, st>>>(d, fail));
  return cudaGetLastError();
}

template <int N>
__global__ void __launch_bounds__(G * N) syev_tiny_kernel(const TinyProb* __restrict__ probs, int* fail) {
  syev_tiny<N>(probs[blockIdx.x], fail);
}

// The descriptors of a call with few blocks, as a kernel parameter: no copy.
struct TinyArgs {
  TinyProb p[TINY_INLINE];
};
template <int N>
__global__ void __launch_bounds__(G * N) syev_tiny_inline_kernel(const __grid_constant__ TinyArgs args, int* fail) {
  syev_tiny<N>(args.p[blockIdx.x], fail);
}

namespace {

template <int N>
cudaError_t tiny_launch(const TinyProb* h, const TinyProb* d, int nprob, int* fail, cudaStream_t st) {
  const int smem = (int)sizeof(TinySm<N>);
  cudaError_t e = d ? cudaFuncSetAttribute(syev_tiny_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
                    : cudaFuncSetAttribute(syev_tiny_inline_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  if (d) {
    NRGB_LAUNCH("syev_small", st, syev_tiny_kernel<N><<<nprob, G * N, smem, st>>>(d, fail));
  } else {
    TinyArgs args;
    for (int i = 0; i < nprob; ++i) args.p[i] = h[i];
    NRGB_LAUNCH("syev_small", st, syev_tiny_inline_kernel<N><<<nprob, G * N, smem, st>>>(args, fail));
  }
  return cudaGetLastError();
}

}  // namespace

// One launch, for the largest block: a CTA for up to 32 rows takes 37 KB of shared
// memory, so that 6 share an SM, one for up to 8 rows 4 KB and a single warp.
// Measured (kernel, us; 32 rows for all in brackets; before it a warp a block): 4000
// blocks of 2 to 4 rows 28 (93; 38), of 8 56 (217; 145), of 16 187 (463 before).
cudaError_t syev_tiny_launch(const TinyProb* h, const TinyProb* d, int nprob, int* fail, cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  int nmax = 0;
  for (int i = 0; i < nprob; ++i) nmax = std::max(nmax, h[i].n);
  return nmax <= 8    ? tiny_launch<8>(h, d, nprob, fail, st)
         : nmax <= 16 ? tiny_launch<16>(h, d, nprob, fail, st)
                      : tiny_launch<SYEV_TINY>(h, d, nprob, fail, st);
}

}  // namespace nrgb
