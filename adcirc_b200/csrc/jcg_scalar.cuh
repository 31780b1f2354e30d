// jcg_scalar.cuh -- ITPACK's adaptive eigenvalue estimate (chgcon) by one
// warp, shared by the JCG kernels that give it a warp of its own, and bounds of
// it.
#pragma once

#include "jcg_chgcon.cuh"

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

// zbrent's tolerance.
__device__ inline double zbrent_tol(double zeta) { return pow10_neg(nsig_of(zeta)); }

// 2^-e for 0 <= e < 1000.
__device__ __forceinline__ double pow2_neg(int e) {
  return __longlong_as_double((long long)(1023 - e) << 52);
}

// The largest eigenvalue of the CG tridiagonal in [lo, 1] itself, by one
// warp: 32 points of the bracket are evaluated at once and the sign change
// found by ballot.  The first points cluster around lo + gprev, the step the
// eigenvalue took last time; the next ones, by powers of two, around the root
// of the inverse cubic through the four points about the sign change
// (Neville's scheme, every lane its own stencil).  This takes two rounds, now
// and then three, 2,000 to 2,800 cycles against zbrent's 5,000 to 7,500, and
// stops when the cubic's error bound w (w / (x - lo))^3 is below 1e-14 of the
// root (errors against LAPACK on the systems of the test meshes: 4e-15 at
// most).  Returns an ier as zbrent does (502: no sign change, 501: not found).
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
    if (round == 0) {
      // no value may run out of range beside the root, where zbrent would take
      // it for the root itself (hundreds of rows)
      if (!(rcp_range(flo) && rcp_range(fhi))) return 501;
      if ((flo > 0.0) == (fhi > 0.0)) return 502;
    }
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
// reference writes it, and of the determinant, 250 + 10 n.  kFast: 420, with
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

// (root, ier)
static __device__ __noinline__ double2 zbrent_plain(int n, const double2 *tri, double t, int maxfn, double a) {
  double root = 0.0;
  const int ier = zbrent_by<false>(n, tri, t, maxfn, a, root);
  return make_double2(root, ier);
}

// tri(in, 1) and tri(in, 2), in one division.
__device__ __forceinline__ void tri_entries(double gamma, double rho, double gamold, double rhoold, double2 *tri,
                                            int in) {
  const int lane = threadIdx.x & 31;
  const double num = lane == 0 ? 1.0 : 1.0 - rho;
  const double den = lane == 0 ? gamma : rho * rhoold * gamma * gamold;
  const double q = num / den;
  if (lane == 0) tri[in].x = 1.0 - q;
  if (lane == 1) tri[in - 1].y = q;
  __syncwarp();
}

// chgcon, jacobi case (itpackv.F:893-1027), for iteration `in`; every lane
// of the scalar warp holds the same cme, cmold and adapt.
// gamma and rho are those of parcon(in - 1), gamold and rhoold of the
// iteration before; tol is zbrent_tol(zeta).
// kFast as zbrent_by's (the resident kernel, which seldom runs chgcon, keeps
// its registers for its rows).
template <bool kFast>
__device__ __forceinline__ void chgcon_warp(double gamma, double rho, double gamold, double rhoold, double zeta,
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
  tri_entries(gamma, rho, gamold, rhoold, tri, in);
  double root = 0.0;
  ier = zbrent_by<kFast>(in, tri, tol, max(itmax, 50), start, root);
  if (kFast && ier < 0) {
    const double2 r = zbrent_plain(in, tri, tol, max(itmax, 50), start);
    root = r.x;
    ier = (int)r.y;
  }
  if (ier != 0) {
    adapt = 0;
    return;
  }
  cme = root;
}

// Bounds of chgcon's estimate from the eigenvalue itself, at 2,400 cycles a
// call instead of zbrent's.
//
// While chgcon finds a root in every iteration, the estimate of iteration `in`
// lies within zbrent's tolerance of the eigenvalue lam of the leading rows.  It
// surely finds one while the eigenvalue has grown by more than the tolerances
// and zeta allow for (else it may have stopped: |cme - cmold| <= zeta cme, or
// no sign change because the last point lay beyond the root).  From the first
// iteration for which that is not sure, the estimate is no less than it was
// (it never decreases) and no more than the eigenvalue with the tolerance.
struct CmeBounds {
  double lam, lamp, gprev;    // the eigenvalue, the one before, its last step
  double low, up;
  bool found, sure;

  // After chgcon(0) and chgcon(1), which are exact.
  __device__ __forceinline__ void start(double zeta, double cme0, double cme1) {
    lamp = cme0;
    lam = low = up = cme1;
    gprev = 0.0;
    found = true;
    sure = lam != 0.0 && zeta < 1.0;   // |cme - 0| <= zeta cme
  }
  // Iteration in >= 2, whose rows of tri are set; tol is zbrent_tol(zeta).
  __device__ __forceinline__ void next(double zeta, double tol, const double2 *tri, int in) {
    double root = 0.0;
    const double margin = in == 2 ? 0.0 : tol * fmax(fabs(lam), 0.1) * 1.001 + 1.0e-13;
    const bool ok = found && tri_root_warp(in, tri, lam - margin, gprev, root) == 0 && root >= lam && root < 1.0;
    if (!ok) {
      found = sure = false;
      up = INFINITY;
      return;
    }
    const double tb = tol * fmax(root, 0.1) * 1.001 + 1.0e-13;
    sure = sure && root > lam + margin && (in == 2 || lam - lamp > zeta * fabs(lam) + 2.0 * tb);
    if (sure) low = root - tb;
    up = root + tb;
    gprev = root - lam;
    lamp = lam;
    lam = root;
  }
};

}  // namespace adc
