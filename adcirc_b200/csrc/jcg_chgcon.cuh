// jcg_chgcon.cuh -- ITPACK's adaptive eigenvalue estimate (chgcon) as the
// reference runs it, on one thread: in jcg_kernel's scalar block, and on the
// host for the solves whose stopping test needed bounds only.
#pragma once

#include "adc_internal.cuh"

#include <algorithm>
#include <cmath>

namespace adc {

// Serial ITPACK state of one solve, held in registers of the scalar block's
// thread 0 (echall/itjcg/chgcon/pstop/parcon variables).
struct ItpLocal {
  double zeta, cme, gamma, rho, gamold, rhoold, delnnm, delsnm, udnm, stptst, cmold, rparm1;
  int itmax, adapt, q1, isym, chg_ier;
};

// ---------------------------------------------------------------- scalars
// determ (itpackv.F:1029-1068): the three-term recurrence for
// det(tri - x I), evaluated with the two trailing values in registers
// (same operations, same order as the wk1/wk2 arrays of the reference).
// tri(i,1) = t1[i-1], tri(i,2) = t2[i-1], held in shared memory.
__host__ __device__ inline double determ_d(int n, const double *t1, const double *t2, double xlmda) {
  double w2 = t1[n - 1] - xlmda;                       // wk2(n)
  double w1 = (t1[n - 2] - xlmda) * w2 + t2[n - 1];    // wk2(n-1)
  for (int l = n - 2; l >= 1; --l) {
    double w = (t1[l - 1] - xlmda) * w1 + t2[l] * w2;  // wk2(l)
    w2 = w1;
    w1 = w;
  }
  return w1;
}

// zbrent (itpackv.F:2521-2781): Brent root of the characteristic
// polynomial of the CG tridiagonal on [a, b].
__host__ __device__ inline void zbrent_d(int n, const double *t1, const double *t2, double eps, double t,
                         double &a, double &b, int &maxfn, int &ier) {
  double c = 0, d = 0, e = 0, p, q, r, s, fa, fb, fc, tol, rm, rone, temp;
  ier = 0;
  int ic = 2;
  fa = determ_d(n, t1, t2, a);
  fb = determ_d(n, t1, t2, b);
  s = b;
  if ((fa > 0.0 && fb > 0.0) || (fa < 0.0 && fb < 0.0)) {
    ier = 502;
    maxfn = ic;
    return;
  }
  bool reset = true;
  for (;;) {
    if (reset) {
      c = a;
      fc = fa;
      d = b - c;
      e = d;
    }
    reset = false;
    if (!(fabs(fc) >= fabs(fb))) {
      a = b; b = c; c = a;
      fa = fb; fb = fc; fc = fa;
    }
    tol = t * fmax(fabs(b), 0.1);
    rm = (c - b) * 0.5;
    if (fabs(fb) <= eps || fabs(c - b) <= tol) {
      a = c;
      maxfn = ic;
      return;
    }
    if (ic >= maxfn) {
      ier = 501;
      a = c;
      maxfn = ic;
      return;
    }
    bool bisect = false;
    if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
      bisect = true;
    } else {
      s = fb / fa;
      if (a == c) {
        p = (c - b) * s;
        q = 1.0 - s;
      } else {
        q = fa / fc;
        r = fb / fc;
        rone = r - 1.0;
        p = s * ((c - b) * q * (q - r) - (b - a) * rone);
        q = (q - 1.0) * rone * (s - 1.0);
      }
      if (p > 0.0) q = -q;
      if (p < 0.0) p = -p;
      s = e;
      e = d;
      if (p + p >= 3.0 * rm * q || p + p >= fabs(s * q)) {
        bisect = true;
      } else {
        d = p / q;
      }
    }
    if (bisect) {
      e = rm;
      d = e;
    }
    a = b;
    fa = fb;
    temp = d;
    if (fabs(temp) <= 0.5 * tol) temp = copysign(0.5 * tol, rm);
    b = b + temp;
    s = b;
    fb = determ_d(n, t1, t2, s);
    ic = ic + 1;
    if (fb == 0.0 || fc == 0.0) continue;
    if ((fb > 0.0 && fc < 0.0) || (fb < 0.0 && fc > 0.0)) continue;
    reset = true;
  }
}

// int(-log10(zeta)) as a glibc-linked Fortran build evaluates it: the
// logarithm rounded to the nearest double, then truncated.  Values within
// 1e-12 of an integer are taken as that integer (the correctly rounded
// logarithm of a double nearest a power of ten is that integer).
__host__ __device__ inline int nsig_of(double zeta) {
  double L = -log10(fabs(zeta));
  double k = rint(L);
  int itmp = (fabs(L - k) <= 1e-12 * fmax(1.0, fabs(k))) ? (int)k : (int)L;
  return itmp > 4 ? itmp : 4;
}

__host__ __device__ inline double pow10_neg(int nsig) {
  double p = 1.0;
  for (int i = 0; i < nsig; ++i) p *= 10.0;   // exact up to 1e22
  return 1.0 / p;
}

// chgcon, jacobi case (itpackv.F:893-1027), for iteration `in`.  The
// tridiagonal is t1, t2.
__host__ __device__ inline void chgcon_d(ItpLocal *it, double *t1, double *t2, int in) {
  double start = it->cme, end1 = 0.0;
  int ip = in;
  if (ip == 0) {
    it->cmold = 0.0;
    it->cme = 0.0;
    return;
  }
  if (ip == 1) {
    end1 = 1.0 - 1.0 / it->gamma;
    t1[0] = end1;
    t2[0] = 0.0;
    it->cme = end1;
    return;
  }
  if (fabs(start - it->cmold) <= it->zeta * start) {
    it->adapt = 0;
    return;
  }
  it->cmold = start;
  t1[ip - 1] = 1.0 - 1.0 / it->gamma;
  t2[ip - 1] = (1.0 - it->rho) / (it->rho * it->rhoold * it->gamma * it->gamold);
  int ier = 0;
  if (it->isym != 0) {
    ier = 903;
  } else {
    int nsig = nsig_of(it->zeta);
    int maxfn = it->itmax > 50 ? it->itmax : 50;
    double a = start, b = 1.0;
    zbrent_d(ip, t1, t2, 0.0, pow10_neg(nsig), a, b, maxfn, ier);
    end1 = b;
  }
  it->chg_ier = ier;
  if (ier != 0) {
    it->adapt = 0;
    return;
  }
  it->cme = end1;
}

}  // namespace adc
