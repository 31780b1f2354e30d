// jcg_scalar.cuh -- ITPACK's adaptive eigenvalue estimate (chgcon) by one
// warp, shared by the JCG kernels that give it a warp of its own.
#pragma once

#include "adc_internal.cuh"

#include <cfloat>

namespace adc {

// The CG tridiagonal as determ reads it: p[l] = (tri(l,1), tri(l+1,2)).
// det(tri - x I) by its three-term recurrence (itpackv.F:1029-1068), with
// one fused multiply-add per term on the dependent chain.
__device__ __forceinline__ double tri_det(int n, const double2 *p, double x) {
  double w2 = p[n].x - x;
  double w1 = fma(p[n - 1].x - x, w2, p[n - 1].y);
  const double2 q3 = p[3], q2 = p[2], q1 = p[1];   // the last terms, requested at the start
  int l = n - 2;
#pragma unroll 2
  for (; l >= 4; l -= 4) {
    const double2 a = p[l], b = p[l - 1], c = p[l - 2], d = p[l - 3];
    w2 = fma(a.x - x, w1, a.y * w2);
    w1 = fma(b.x - x, w2, b.y * w1);
    w2 = fma(c.x - x, w1, c.y * w2);
    w1 = fma(d.x - x, w2, d.y * w1);
  }
  if (l >= 3) {
    const double w = fma(q3.x - x, w1, q3.y * w2);
    w2 = w1;
    w1 = w;
  }
  if (l >= 2) {
    const double w = fma(q2.x - x, w1, q2.y * w2);
    w2 = w1;
    w1 = w;
  }
  if (l >= 1) w1 = fma(q1.x - x, w1, q1.y * w2);
  return w1;
}

// 1/x to a few ulp for |x| well inside the normal range: the hardware's
// approximation and two Newton steps, without a division's range checks.
__device__ __forceinline__ double rcp_estimate(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

// 2^-e for 0 <= e < 1000.
__device__ __forceinline__ double pow2_neg(int e) {
  return __longlong_as_double((long long)(1023 - e) << 52);
}

// The largest eigenvalue of the CG tridiagonal in [lo, 1] (zbrent's role,
// itpackv.F:2521-2781), by one warp: 32 points of the bracket are evaluated
// at once and the sign change found by ballot.  The first points cluster
// around lo + gprev, the step the estimate took last time; the next ones, by
// powers of two, around the root of the inverse cubic through the four
// points about the sign change (Neville's scheme, every lane its own
// stencil).  The reference's Brent search takes about eight determinants and
// as many chains of divisions one after another: 9,700 to 18,000 cycles a
// call here, more than the rest of an iteration on meshes up to 100k nodes.
// This takes two rounds, now and then three, and stops when the cubic's
// error bound w (w / (x - lo))^3 is below 1e-14 of the root, well under
// zbrent's own tolerance of 10^-nsig (errors against LAPACK on the systems
// of the test meshes: 4e-15 at most).  Returns zbrent's ier (502: no sign
// change, 501: not found).
__device__ inline int tri_root_warp(int n, const double2 *tri, double lo, double gprev, double &root) {
  const int lane = threadIdx.x & 31;
  const double span = 1.0 - lo;
  double x;
  {
    // lanes 1-24: lo + g 2^((lane - 14) / 4); lanes 25-30 close in on 1
    const double g = gprev > 0.0 ? fmin(gprev, 0.5 * span) : 0.25 * span;
    const double f4[4] = {1.0, 1.189207115002721, 1.4142135623730951, 1.681792830507429};
    const int e4 = min(max(lane, 1), 24) + 2;   // lane - 14 = e4 - 16
    const double sc = (e4 >> 2) >= 4 ? (double)(1 << ((e4 >> 2) - 4)) : pow2_neg(4 - (e4 >> 2));
    x = fmin(lo + g * (sc * f4[e4 & 3]), 1.0);
    const double top = __shfl_sync(0xffffffffu, x, 24);
    if (lane > 24) x = top + (1.0 - top) * pow2_neg(2 * (31 - lane));
    if (lane == 0) x = lo;
    if (lane == 31) x = 1.0;
  }
  for (int round = 0; round < 60; ++round) {
    const double f = tri_det(n, tri, x);
    const double flo = __shfl_sync(0xffffffffu, f, 0), fhi = __shfl_sync(0xffffffffu, f, 31);
    if (round == 0 && ((flo > 0.0 && fhi > 0.0) || (flo < 0.0 && fhi < 0.0))) return 502;
    const bool hit = f == 0.0 || (fhi > 0.0 ? f > 0.0 : f < 0.0);
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (m & 1u) {   // the lower end itself is the root
      root = __shfl_sync(0xffffffffu, x, 0);
      return 0;
    }
    if (m == 0) return 501;
    const int k = __ffs(m) - 1;
    // inverse cubic at f = 0 through points i .. i + 3 of every lane i; the
    // three divisors are inverted side by side (true divisions took 200 to
    // 500 cycles each here).  Stencils with equal values (coinciding points,
    // the last lanes) give no number and fail the test below.
    double P = x, F[3], rd[3];
#pragma unroll
    for (int lev = 0; lev < 3; ++lev) {
      F[lev] = __shfl_down_sync(0xffffffffu, f, lev + 1);
      rd[lev] = rcp_estimate(F[lev] - f);
    }
#pragma unroll
    for (int lev = 0; lev < 3; ++lev) {
      const double P1 = __shfl_down_sync(0xffffffffu, P, 1);
      P = (P * F[lev] - P1 * f) * rd[lev];
    }
    const double a = __shfl_sync(0xffffffffu, x, k - 1), b = __shfl_sync(0xffffffffu, x, k);
    const double fb = __shfl_sync(0xffffffffu, f, k);
    double xh = __shfl_sync(0xffffffffu, P, min(max(k - 2, 0), 28));
    const double w = b - a;
    if (fb == 0.0 || w <= 4.0 * DBL_EPSILON * fabs(b)) {
      root = b;
      return 0;
    }
    if (!(xh > a && xh < b)) {
      xh = a + 0.5 * w;
    } else {
      const double gap = xh - lo;
      if (w * w * w * w <= 1.0e-14 * fmax(fabs(xh), 0.1) * (gap * gap * gap)) {
        root = xh;
        return 0;
      }
    }
    x = lane < 16 ? xh - (xh - a) * pow2_neg(lane) : xh + (b - xh) * pow2_neg(31 - lane);
    if (lane == 0) x = a;
    if (lane == 31) x = b;
  }
  return 501;
}

// chgcon, jacobi case (itpackv.F:893-1027), for iteration `in`; every lane
// of the scalar warp holds the same cme, cmold and adapt.
// gamma and rho are those of parcon(in - 1), gamold and rhoold of the
// iteration before.
__device__ inline void chgcon_warp(double gamma, double rho, double gamold, double rhoold, double zeta,
                                   double2 *tri, int in, double &cme, double &cmold, double &gprev,
                                   int &adapt, int &ier) {
  if (in == 0) {
    cmold = 0.0;
    cme = 0.0;
    return;
  }
  const int lane = threadIdx.x & 31;
  if (in == 1) {
    cme = 1.0 - 1.0 / gamma;
    if (lane == 0) {
      tri[1].x = cme;
      tri[0].y = 0.0;
    }
    __syncwarp();
    return;
  }
  const double start = cme;
  if (fabs(start - cmold) <= zeta * start) {
    adapt = 0;
    return;
  }
  cmold = start;
  {
    // lane 0: tri(in, 1), the others: tri(in, 2), in one division
    const double num = lane == 0 ? 1.0 : 1.0 - rho;
    const double den = lane == 0 ? gamma : rho * rhoold * gamma * gamold;
    const double q = num / den;
    if (lane == 0) tri[in].x = 1.0 - q;
    if (lane == 1) tri[in - 1].y = q;
  }
  __syncwarp();
  double root = 0.0;
  ier = tri_root_warp(in, tri, start, gprev, root);
  if (ier != 0) {
    adapt = 0;
    return;
  }
  gprev = root - start;
  cme = root;
}

}  // namespace adc
