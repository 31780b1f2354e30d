// jcg_scalar.cuh -- ITPACK's adaptive eigenvalue estimate (chgcon) by one
// warp, shared by the JCG kernels that give it a warp of its own.
#pragma once

#include "adc_internal.cuh"

#include <cfloat>

namespace adc {

// The CG tridiagonal as determ reads it: p[l] = (tri(l,1), tri(l+1,2)).
// det(tri - x I) by its three-term recurrence (itpackv.F:1029-1068), with
// one fused multiply-add per term on the dependent chain.  Four rows at a
// time, the next four requested before; rows past the last one multiply by one
// (a loop over the remainder took 200 cycles).
__device__ __forceinline__ double tri_det(int n, const double2 *p, double x) {
  double w2 = 0.0, w1 = 1.0;
  int l = (n + 3) & ~3;
  double2 r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = p[min(l - k, n)];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double c = l - k > n ? 1.0 : r[k].x - x, y = l - k >= n ? 0.0 : r[k].y;
    const double w = fma(c, w1, y * w2);
    w2 = w1;
    w1 = w;
  }
#pragma unroll 2
  for (l -= 4; l > 0; l -= 4) {
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = p[l - k];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double w = fma(r[k].x - x, w1, r[k].y * w2);
      w2 = w1;
      w1 = w;
    }
  }
  return w1;
}

// 1/x to a few ulp for |x| between 2^-900 and 2^900: the hardware's
// approximation and two Newton steps, without a division's range checks.
__device__ __forceinline__ double rcp_estimate(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}
__device__ __forceinline__ bool rcp_range(double x) {
  return (unsigned)((__double2hiint(x) & 0x7fffffff) - ((1023 - 900) << 20)) < (unsigned)(1800 << 20);
}

// |x| as an integer that orders like it.
__device__ __forceinline__ long long mag(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }

// zbrent's tolerance 10^-nsig, nsig = max(4, int(-log10(zeta))), with the
// logarithm as a glibc-linked Fortran build evaluates it: rounded to the
// nearest double, then truncated.  Values within 1e-12 of an integer are taken
// as that integer (the correctly rounded logarithm of a double nearest a power
// of ten is that integer).
__device__ inline double zbrent_tol(double zeta) {
  const double L = -log10(fabs(zeta)), k = rint(L);
  const int itmp = fabs(L - k) <= 1e-12 * fmax(1.0, fabs(k)) ? (int)k : (int)L;
  double p = 1.0;
  for (int i = 0; i < max(itmp, 4); ++i) p *= 10.0;   // exact up to 1e22
  return 1.0 / p;
}

// zbrent (itpackv.F:2521-2781): Brent's search for the largest eigenvalue of
// the CG tridiagonal in [a, 1], to the tolerance t; returns its ier (502: no
// sign change, 501: not found in maxfn determinants).  The estimate that
// ITPACK goes on with is the search's last point, which lies within the
// tolerance of the eigenvalue and not at it: with zeta at 1e-5 a search that
// finds the eigenvalue itself stops solves of ill-conditioned systems up to
// six iterations earlier or later.  So the steps are zbrent's, one after
// another, and every lane takes them.
//
// What bounds a step is the latency of its serial logic, 600 cycles as the
// reference writes it, and of the determinant, 60 + 10 n.  kFast: 420, with
// multiplications by reciprocals formed as soon as a value is there, both
// interpolations side by side, selections for branches and comparisons of
// integers; it gives up (-1) on values that have no such reciprocal.
template <bool kFast>
__device__ __forceinline__ int zbrent_by(int n, const double2 *tri, double t, int maxfn, double a, double &root) {
  const auto recip = [](double v) { return kFast ? rcp_estimate(v) : 0.0; };
  const auto over = [](double v, double w, double rw) { return kFast ? v * rw : v / w; };
  double b = 1.0;
  const double f = tri_det(n, tri, (threadIdx.x & 31) ? b : a);
  double fa = __shfl_sync(0xffffffffu, f, 0), fb = __shfl_sync(0xffffffffu, f, 1);
  if ((fa > 0.0 && fb > 0.0) || (fa < 0.0 && fb < 0.0)) return 502;
  if (kFast && !(rcp_range(fa) && rcp_range(fb))) return -1;
  double ra = recip(fa), rb = recip(fb);
  double c = a, fc = fa, rc = ra, d = b - c, e = d;
#pragma unroll 1
  for (int ic = 2;; ++ic) {
    if (mag(fc) < mag(fb)) {
      a = b; b = c; c = a;
      fa = fb; fb = fc; fc = fa;
      ra = rb; rb = rc; rc = ra;
    }
    const double cb = c - b, rm = cb * 0.5;
    const double ht = 0.5 * t * (mag(b) > mag(0.1) ? fabs(b) : 0.1);   // half zbrent's tol
    if (mag(fb) == 0 || mag(rm) <= mag(ht)) {
      root = b;
      return 0;
    }
    if (ic >= maxfn) return 501;
    // the step p/q: the secant's, or inverse quadratic interpolation's
    const double s = over(fb, fa, ra), u = over(fa, fc, rc), r = over(fb, fc, rc), rone = r - 1.0;
    const double pi = s * (cb * u * (u - r) - (b - a) * rone), qi = (u - 1.0) * rone * (s - 1.0);
    const bool sec = a == c;
    const double p = sec ? cb * s : pi, q = sec ? 1.0 - s : qi, w = p > 0.0 ? -q : q;
    const double x = over(fabs(p), w, recip(w)), ax = fabs(x) + fabs(x);
    // taken where it goes less than 3/4 of the way to c and less than half the step before the last
    const bool bisect = ((__double2hiint(x) ^ __double2hiint(rm)) < 0) | (mag(ax) >= mag(3.0 * rm)) |
                        (mag(ax) >= mag(e)) | (mag(e) < mag(ht + ht)) | (mag(fa) <= mag(fb));
    e = bisect ? rm : d;
    d = bisect ? rm : x;
    a = b;
    fa = fb;
    ra = rb;
    b = b + (mag(d) <= mag(ht) ? copysign(ht, rm) : d);
    fb = tri_det(n, tri, b);
    if (kFast && !rcp_range(fb)) {
      if (fb != 0.0) return -1;
    }
    rb = recip(fb);
    if (!(mag(fb) == 0 || mag(fc) == 0 || (__double2hiint(fb) ^ __double2hiint(fc)) < 0)) {
      c = a;
      fc = fa;
      rc = ra;
      d = b - c;
      e = d;
    }
  }
}

static __device__ __noinline__ int zbrent_plain(int n, const double2 *tri, double t, int maxfn, double a, double *root) {
  double r = 0.0;
  const int ier = zbrent_by<false>(n, tri, t, maxfn, a, r);
  *root = r;
  return ier;
}

// chgcon, jacobi case (itpackv.F:893-1027), for iteration `in`; every lane
// of the scalar warp holds the same cme, cmold and adapt.
// gamma and rho are those of parcon(in - 1), gamold and rhoold of the
// iteration before; tol is zbrent_tol(zeta).
__device__ inline void chgcon_warp(double gamma, double rho, double gamold, double rhoold, double zeta,
                                   double tol, int itmax, double2 *tri, int in, double &cme, double &cmold,
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
  ier = zbrent_by<true>(in, tri, tol, max(itmax, 50), start, root);
  if (ier < 0) ier = zbrent_plain(in, tri, tol, max(itmax, 50), start, &root);
  if (ier != 0) {
    adapt = 0;
    return;
  }
  cme = root;
}

}  // namespace adc
