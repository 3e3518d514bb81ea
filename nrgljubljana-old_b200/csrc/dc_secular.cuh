// The secular equation of a rank-one merge, 1 + rho sum_i z_i^2 / (d_i - x) = 0,
// solved by a group of G lanes of a warp per root (shared by the merges inside
// one CTA, dc_base.cu, and those of larger nodes, syev.cu).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace nrgb {
namespace {

// Reciprocal from the hardware's approximation by two Newton steps
// r <- r + r (1 - x r): within an ulp for |x| in [2^-1000, 2^1000], which the
// scaled problems below stay in: values are near 1, and poles that were not
// deflated are at least 8 units of 2^-52 apart.  Not a number for 0, subnormal and
// infinite x: of the callers only the quadratics' coefficients (s, c, cc, qq) can
// vanish, and a root that is not a number fails the test of its bracket, after
// which the other root or the bracket's middle is taken.  On B200 68 cycles (with
// an add) and 16 issue cycles a warp, where a division takes 148 and 65.
__device__ __forceinline__ double rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

// Power of two that brings x near 1 (1 for 0 and for what is not finite).
__device__ __forceinline__ double scale_near_one(double x) {
  if (!(x > 0.0) || !(x <= 1e300)) return 1.0;
  const int ex = min(max(ilogb(x), -1000), 1000);
  return ldexp(1.0, -ex);
}

template <int G>
__device__ __forceinline__ double group_sum(double x) {
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Root j of k poles d (ascending, scaled near 1) with weights z: its distance
// tout from the nearer pole d[oout].  Lane h of the group; every lane of the warp
// calls it, those with on = false idle.  The sum is split after pole `l`: for
// an inner root its left neighbour, for the last root (beyond every pole, below
// d[k-1] + rho |z|^2) the last pole but one.  The first guess solves the equation
// with the poles beyond l and l + 1 frozen at the middle of the root's interval;
// the iteration keeps the values and slopes of both parts (two-pole model)
// inside a bracket.  About 3 iterations, 6 at most in most nodes (the last root
// took 10 with one pole in its model).  bad: not converged, or not a number.
template <int G>
__device__ __forceinline__ void secular_root(const double* d, const double* z, int k, int j, double rho, int h, bool on,
                                             double& tout, int& oout, bool& bad) {
  constexpr double EPS_ = 2.220446049250313e-16;
  bad = false;
  if (k == 1) {  // uniform in the group; such a node's entries run no loop below
    tout = on ? rho * z[0] * z[0] : 0.0;
    oout = 0;
    bad = on && !(fabs(tout) <= 1e300);
    on = false;
  }
  const bool inner = j < k - 1;
  const int l = on ? (inner ? j : k - 2) : 0, r = on ? l + 1 : 0;
  const double dl = on ? d[l] : 0.0, dr = on ? d[r] : 0.0, gap = dr - dl;
  int o = r;
  double tlo = 0.0, thi = 0.0, t = 0.0;
  {
    double zz = 0.0;
    if (on && !inner)
      for (int i = h; i < k; i += G) zz = fma(z[i], z[i], zz);
    zz = group_sum<G>(zz);
    // the middle of the interval, from d[l] (inner) or d[r] (last)
    const double mid = inner ? 0.5 * gap : 0.5 * rho * zz, base = inner ? dl : dr;
    double f = 0.0;
    if (on)
#pragma unroll 4
      for (int i = h; i < k; i += G) {
        const double w = (i == l || i == r) ? 0.0 : z[i] * z[i];
        f = fma(w, rcp_newton(w == 0.0 ? 1.0 : (d[i] - base) - mid), f);
      }
    const double c = fma(rho, group_sum<G>(f), 1.0);
    if (on) {
      const double a = rho * z[l] * z[l], b = rho * z[r] * z[r];
      const bool left = inner && fma(b - a, rcp_newton(mid), c) >= 0.0;  // the equation at the midpoint
      // c t^2 + p t + q = 0 from the pole at hand
      const double p = left ? -(c * gap + a + b) : c * gap - a - b, q = left ? a * gap : -b * gap;
      const double sq = sqrt(fmax(p * p - 4.0 * c * q, 0.0));
      const double s = p >= 0.0 ? -(p + sq) : sq - p;  // roots s / 2c and 2q / s
      o = left ? l : r;
      tlo = inner && !left ? -mid : 0.0;
      thi = inner ? (left ? mid : 0.0) : rho * zz;
      const double r1 = 2.0 * q * rcp_newton(s), r2 = 0.5 * s * rcp_newton(c);
      t = (r1 > tlo && r1 < thi) ? r1 : r2;
      if (!(t > tlo && t < thi)) t = 0.5 * (tlo + thi);
    }
  }
  const double dorig = on ? d[o] : 0.0, dL = dl - dorig, dR = dr - dorig;
  bool done = !on;
  for (int it = 0; it < 400; ++it) {
    if (!__any_sync(0xffffffffu, !done)) break;
    double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
    if (!done) {
      // one loop for both parts: the roots of a warp differ in l
#pragma unroll 4
      for (int i = h; i < k; i += G) {
        const double zi = z[i], q = zi * rcp_newton((d[i] - dorig) - t);
        const double zl = i <= l ? q : 0.0, zr = i <= l ? 0.0 : q;
        psi = fma(zi, zl, psi);
        dpsi = fma(q, zl, dpsi);
        phi = fma(zi, zr, phi);
        dphi = fma(q, zr, dphi);
      }
    }
    psi = group_sum<G>(psi);
    dpsi = group_sum<G>(dpsi);
    phi = group_sum<G>(phi);
    dphi = group_sum<G>(dphi);
    if (done) continue;
    // the group's lanes hold identical sums and run the same scalar update
    const double f = fma(rho, psi + phi, 1.0);
    if (!(fabs(f) <= 1e300)) bad = true;
    if (f == 0.0) {
      done = true;
      continue;
    }
    if (f < 0.0) tlo = t;
    else thi = t;
    const double DL = dL - t, DR = dR - t, uL = rho * dpsi * DL, uR = rho * dphi * DR;
    const double cc = f - uL - uR;
    const double bb = fma(cc, DL + DR, fma(uL, DL, uR * DR));
    const double c0 = DL * DR * f;
    const double sq = sqrt(fmax(fma(bb, bb, -4.0 * cc * c0), 0.0));
    const double qq = (bb >= 0.0) ? bb + sq : bb - sq;
    const double t1 = fma(0.5 * qq, rcp_newton(cc), t), t2 = fma(2.0 * c0, rcp_newton(qq), t);
    double tn = (t2 > tlo && t2 < thi) ? t2 : t1;
    const double terms = rho * (fabs(psi) + fabs(phi));
    if (fabs(tn - t) <= 2.0 * EPS_ * fabs(t) || fabs(f) <= EPS_ * (8.0 + 8.0 * terms)) {
      done = true;
      continue;
    }
    if (!(tn > tlo && tn < thi)) tn = 0.5 * (tlo + thi);
    done = thi - tlo <= 4.0 * EPS_ * fmax(fabs(tlo), fabs(thi));
    t = tn;
  }
  if (on) {
    tout = t;
    oout = o;
    bad = bad || (!done && !(thi - tlo <= 1e-10 * fmax(fabs(tlo), fabs(thi))));
  }
}

// prod_j (lambda_j - d_i) / (d_j' - d_i) of the Loewner formula over this lane's
// j = h, h + G, .. < k - 1, numerators and denominators multiplied in fours
// (scaled differences: no under- or overflow) before one reciprocal.
template <int G>
__device__ __forceinline__ double lowner_product(const double* d, const int* orig, const double* tau, int k, int i, int h) {
  const double di = d[i];
  double prod = 1.0;
  int j = h;
  for (; j + 3 * G < k - 1; j += 4 * G) {
    double num = 1.0, den = 1.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q = j + u * G;
      num *= (d[orig[q]] - di) + tau[q];
      den *= d[q + (q < i ? 0 : 1)] - di;
    }
    prod *= num * rcp_newton(den);
  }
  for (; j < k - 1; j += G) prod *= ((d[orig[j]] - di) + tau[j]) * rcp_newton(d[j + (j < i ? 0 : 1)] - di);
  return prod;
}

}  // namespace
}  // namespace nrgb
