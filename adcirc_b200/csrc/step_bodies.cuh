// step_bodies.cuh -- the 2DDI step (timestep.F, gwce.F, wetdry.F,
// momentum.F, nws08.F90) item by item: what one node, element, boundary entry
// or warp of elements does in each pass.  The kernels (gwce.cu, flux.cu,
// wetdry.cu, momentum.cu) run a pass over the mesh.  Every pass keeps the
// reference's operations and, per node, its element order.
#pragma once

#include "adc_internal.cuh"

#include <cfloat>
#include <cmath>

namespace adc {

// --------------------------------------------------------------- shift
// timestep.F:231-237 (IT==1 H init), :375-416 (time-level shift, zeroing),
// nodalattr.F:2399-2413 (quadratic/linear/hybrid friction), :2700-2704.
// `whole`: the rest of the step follows, so load vectors that it writes
// before anyone reads them are not zeroed; `met_follows`: the vortex forcing
// writes WSX2, WSY2 and PR2 next.
__device__ __forceinline__ void node_shift(const adc_ctx &c, const adc_step_t &st, int i, bool whole,
                                           bool met_follows) {
  const adc_params_t &p = c.p;
  if (st.it == 1) {
    double h = c.dp[i] + p.ifnlfa * c.eta2[i];
    c.h2[i] = h;
    c.h1[i] = h;
  }
  c.qx1[i] = c.qx2[i];
  c.qy1[i] = c.qy2[i];
  double u1 = c.uu2[i], v1 = c.vv2[i];
  c.uu1[i] = u1;
  c.vv1[i] = v1;
  if (!whole) {
    c.gwce_lv[i] = 0.0;
    c.mom_x[i] = 0.0;
    c.mom_y[i] = 0.0;
  }
  if (p.nws != 0) {
    c.wsx1[i] = c.wsx2[i];
    c.wsy1[i] = c.wsy2[i];
    c.pr1[i] = c.pr2[i];
  }
  if (!met_follows) {
    if (p.nws != 0) {
      c.wsx2[i] = 0.0;
      c.wsy2[i] = 0.0;
    }
    c.pr2[i] = p.prbckgrnd_mh2o;
  }
  double uv1 = sqrt(u1 * u1 + v1 * v1);
  double h1 = c.dp[i] + p.ifnlfa * c.eta2[i];
  double hyb = 0.0;
  if (p.ifhybf != 0) hyb = p.ifhybf * pow(1.0 + pow(p.hbreak / h1, p.ftheta), p.fgamma / p.ftheta);
  double v = c.fric[i] * (p.iflinbf + (uv1 / h1) * (p.ifnlbf + hyb));
  double cap = 2.0 / p.dt;
  double tk = (v < cap) ? v : cap;
  c.tk[i] = tk;
  c.tkm[3 * i + 0] = tk;
  c.tkm[3 * i + 1] = tk;
  c.tkm[3 * i + 2] = 0.0;
  if (c.nfluxib) c.nib[i] = 0;   // NIBNODECODE(:) = 0, timestep.F:1004
}

// ----------------------------------------------------------------- met
constexpr double kE = 2.718281828459045;       // constants.F90:76
constexpr double kOne2Ten = 0.8928;            // constants.F90:105
constexpr double kPrBckgrndMb = 1013.0;        // constants.F90:55
constexpr double kRhoWat0 = 1000.0;            // constants.F90:49

// GetHollandStormData (nws08.F90:827-878) and the per-storm part of
// HollandGet (nws08.F90:602-639): the state of this step from that of the
// last.  The position is interpolated with the WTRATIO left by the previous
// call, as the reference does.
// Returns whether the time is past the end of the track.
__device__ inline bool vortex_advance(const adc_ctx &c, double timeloc, VortexState &v) {
  bool past = false;
  const adc_vortex_fix_t *f = c.vfix;
  int i = v.counter;
  if (timeloc > f[i].time) {
    i = i + 1;
    if (i >= c.vpar.nfix) {   // nws08.F90:847-852: past the end of the track
      v.err = 1;
      past = true;
      i = c.vpar.nfix - 1;
    }
  }
  const double lon = f[i - 1].x + v.wtratio * (f[i].x - f[i - 1].x);
  const double lat = f[i - 1].y + v.wtratio * (f[i].y - f[i - 1].y);
  v.counter = i;
  if (f[i].cpress < 0.0 || f[i - 1].cpress < 0.0) {
    // a CALM line on either side (nws08.F90:858-872): no storm, WTRATIO kept
    v.calm = 1;
    v.x = lon;
    v.y = lat;
    return past;
  }
  v.calm = 0;
  const double wt = (timeloc - f[i - 1].time) / (f[i].time - f[i - 1].time);
  v.wtratio = wt;
  const double cpress = f[i - 1].cpress + wt * (f[i].cpress - f[i - 1].cpress);
  double spd = f[i - 1].vmax + wt * (f[i].vmax - f[i - 1].vmax);
  const double rmw = f[i - 1].rmw + wt * (f[i].rmw - f[i - 1].rmw);
  const double tvx = f[i - 1].tvx + wt * (f[i].tvx - f[i - 1].tvx);
  const double tvy = f[i - 1].tvy + wt * (f[i].tvy - f[i - 1].tvy);
  // HollandGet: pressure deficit floor, translation removal, BL adjustment,
  // the limited Holland B (backgroundWindFac = 1 for the radial-velocity-
  // weighted background model, nws08.F90:480-485)
  double dpdef = kPrBckgrndMb * 100.0 - cpress;
  if (dpdef < 100.0) dpdef = 100.0;
  const double ts = sqrt(tvx * tvx + tvy * tvy);
  spd = spd - 1.0 * ts;
  spd = spd / c.vpar.bladj;
  double b = c.vpar.rho_air * kE * (spd * spd) / dpdef;
  if (b < 1.0) b = 1.0;
  if (b > 2.5) b = 2.5;
  v.x = lon;
  v.y = lat;
  v.cpress = cpress;
  v.dpdef = dpdef;
  v.spd = spd;
  v.b = b;
  v.rmw = rmw * 1000.0;
  v.tvx = tvx;
  v.tvy = tvy;
  return past;
}

// The node loop of HollandGet (nws08.F90:642-715) followed by the NWS = 8
// stress and pressure of wind.F:1172-1198 (capped Garratt drag,
// wind.F:514-539; no directional reduction, canopy or ice).
__device__ __forceinline__ void node_vortex(const adc_ctx &c, const VortexState &v, double rampmete, int i) {
  double wx, wy, prn2;
  if (v.calm) {   // HollandGet's CALM return (nws08.F90:588-601)
    wx = 0.0;
    wy = 0.0;
    prn2 = kPrBckgrndMb * 100.0 / (kRhoWat0 * c.p.g);
  } else {
    const double hemi = c.vpar.hemisphere >= 0 ? 1.0 : -1.0;   // sign(1, lat)
    const double dx = c.x[i] - v.x;
    const double dy = c.y[i] - v.y;
    const double theta = atan2(dy, dx);
    const double rad = sqrt(dx * dx + dy * dy);
    const double f = c.corif[i];
    const double alpha = pow(v.rmw / rad, v.b);
    double press = v.cpress + v.dpdef * exp(-alpha);
    double vr = sqrt(alpha * exp(1.0 - alpha) * v.spd * (v.spd + 0.0) + 0.25 * (rad * rad) * (f * f)) -
                0.5 * rad * fabs(f);
    vr = vr * c.vpar.wind_mult;
    vr = vr * c.vpar.bladj;
    // inflow angle 0 (useInflow = .false.): theta + sign(1,lat)*0 == theta
    wx = (-hemi) * vr * sin(theta + hemi * 0.0);
    wy = hemi * vr * cos(theta + hemi * 0.0);
    // calcTranslationSpeed, radial-velocity-weighted (nws08.F90:746-749)
    const double tsx = (fabs(vr) / v.spd) * v.tvx;
    const double tsy = (fabs(vr) / v.spd) * v.tvy;
    wx = wx + tsx;
    wy = wy + tsy;
    if (c.vpar.avg_minute == 1) {
      wx = wx * kOne2Ten;
      wy = wy * kOne2Ten;
    }
    press = fmax(0.85e5, fmin(1.1e5, press));
    wx = fmax(-200.0, fmin(200.0, wx));
    wy = fmax(-200.0, fmin(200.0, wy));
    prn2 = press / (kRhoWat0 * c.p.g);
  }
  // wind.F:1174-1193
  const double mag = sqrt(wx * wx + wy * wy);
  double drag = 0.001 * (0.75 + 0.067 * mag);
  if (drag > c.vpar.drag_limit) drag = c.vpar.drag_limit;
  const double awr = c.vpar.rho_air / kRhoWat0;   // airwaterdensityrat, wind.F:349
  c.wsx2[i] = rampmete * awr * drag * wx * mag;
  c.wsy2[i] = rampmete * awr * drag * wy * mag;
  const double prdiff = rampmete * (prn2 - c.p.prbckgrnd_mh2o);
  c.pr2[i] = c.p.prbckgrnd_mh2o + prdiff;
}

// ----------------------------------------------------------------- LHS
// Moves the COEF drift from a point after the solve to the next step that
// keeps COEF, so steps that rebuild COEF never pay for it.  It repeats the
// exact operations of the solve's scal/unscal pass (itpackv.F:2393-2398,
// 2458-2463) with the w = 1/sqrt(diag) that solve used, so COEF ends with
// the same bits as if the solve had written it.
__device__ __forceinline__ void row_drift(const adc_ctx &c, int i) {
  const double wi = c.jw[i];
  const double winv_i = 1.0 / wi;
  const int s = i / kSlice, lane = i - s * kSlice;
  const int base = c.sl_ptr[s] + lane, len = c.rlen[i];
  // a chunk's loads issue together: two round trips instead of two a slot
  for (int kc = 0; kc < len; kc += kGatherChunk) {
    double wj[kGatherChunk], v[kGatherChunk];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (kc + k < len) {
        const int q = base + (kc + k) * kSlice;
        v[k] = c.offd[q];
        wj[k] = c.jw[c.col[q]];
      }
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (kc + k < len) {
        const double sv = v[k] * wi * wj[k];
        c.offd[base + (kc + k) * kSlice] = sv * winv_i * (1.0 / wj[k]);
      }
  }
}

// gwce.F:456-593: nine consistent-mass + gravity entries per element.
// The entries depend on the element's static geometry and depth and on two
// per-step inputs, NCEle and ALPHAL; an element is recomputed only when
// those differ from the values its cached entries were built with (every
// element on the first rebuild and after a host upload), and the nodes of
// a recomputed element are marked for the row gather.  The cached entries
// equal what a full rebuild writes, bit for bit.
template <class R>
__device__ __forceinline__ void elem_lhs(const adc_ctx &c, int e) {
  int n1 = c.nm[3 * e], n2 = c.nm[3 * e + 1], n3 = c.nm[3 * e + 2];
  int NCEle = c.nodecode[n1] * c.nodecode[n2] * c.nodecode[n3] * c.noff[e];
  const double ald = c.alphal[e];
  if (c.lhs_nc[e] == NCEle &&
      __double_as_longlong(c.lhs_al[e]) == __double_as_longlong(ald))
    return;
  const adc_params_t &p = c.p;
  const R DT = R(p.dt);
  R FDX1 = c.fdx[3 * e], FDX2 = c.fdx[3 * e + 1], FDX3 = c.fdx[3 * e + 2];
  R FDY1 = c.fdy[3 * e], FDY2 = c.fdy[3 * e + 1], FDY3 = c.fdy[3 * e + 2];
  R AreaIE2 = c.areas[e];
  R AreaIE = AreaIE2 * R(0.5);
  R AreaIE4 = AreaIE2 * R(2.0);
  R DPAvg = (c.dp[n1] + c.dp[n2] + c.dp[n3]) / R(3.0);
  R GA = R(ald) * R(p.a00) * R(p.g) * DPAvg / AreaIE4;
  R Tau0Avg = (c.tau0[n1] + c.tau0[n2] + c.tau0[n3]) / R(3.0);
  R MsOn = 2 * AreaIE * (R(1.0) / DT + Tau0Avg / R(2.0)) / DT / R(12.0);
  R MsOff = 1 * AreaIE * (R(1.0) / DT + Tau0Avg / R(2.0)) / DT / R(12.0);
  R nc = (R)NCEle;
  R *o = reinterpret_cast<R *>(c.lhs_ebuf) + 9 * (size_t)e;
  o[0] = (MsOn + GA * (FDX1 * FDX1 + FDY1 * FDY1)) * nc;
  o[1] = (MsOn + GA * (FDX2 * FDX2 + FDY2 * FDY2)) * nc;
  o[2] = (MsOn + GA * (FDX3 * FDX3 + FDY3 * FDY3)) * nc;
  o[3] = (MsOff + GA * (FDX1 * FDX2 + FDY1 * FDY2)) * nc;  // (n1, J12)
  o[4] = (MsOff + GA * (FDX1 * FDX3 + FDY1 * FDY3)) * nc;  // (n1, J13)
  o[5] = (MsOff + GA * (FDX2 * FDX1 + FDY2 * FDY1)) * nc;  // (n2, J21)
  o[6] = (MsOff + GA * (FDX2 * FDX3 + FDY2 * FDY3)) * nc;  // (n2, J23)
  o[7] = (MsOff + GA * (FDX3 * FDX1 + FDY3 * FDY1)) * nc;  // (n3, J31)
  o[8] = (MsOff + GA * (FDX3 * FDX2 + FDY3 * FDY2)) * nc;  // (n3, J32)
  c.lhs_nc[e] = NCEle;
  c.lhs_al[e] = ald;
  c.lhs_dirty[n1] = 1;
  c.lhs_dirty[n2] = 1;
  c.lhs_dirty[n3] = 1;
}

// Per-row gather of COEF in element order; returns diag^2 for EP (gwce.F:
// 646-650).  `all`: every row (else the rows of recomputed elements and those
// the boundary pass rewrites).
template <class R>
__device__ __forceinline__ double row_lhs(const adc_ctx &c, int i, bool all) {
  const R *eb = reinterpret_cast<const R *>(c.lhs_ebuf);
  double d2 = 0.0;
  // rows whose elements did not change keep their gathered off-diagonals;
  // only their diagonal, which each solve's scal/unscal rewrites, returns
  // to the gathered value
  if (!all && !c.lhs_dirty[i] && !c.bc_row[i]) {
    const double d = c.diag_gathered[i];
    c.diag[i] = d;
    d2 = d * d;
  } else {
    R d = R(0.0);
    const int q0 = c.n2e_ptr[i], q1 = c.n2e_ptr[i + 1];
    for (int qc = q0; qc < q1; qc += kGatherChunk) {
      int ek[kGatherChunk];
      R x[kGatherChunk];
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) ek[k] = c.n2e[qc + k];
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k)
        if (qc + k < q1) {
          int e = ek[k] / 3, kk = ek[k] - 3 * e;
          x[k] = eb[9 * (size_t)e + kk];
        }
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) d = d + x[k];
    }
    c.diag[i] = (double)d;
    c.diag_gathered[i] = (double)d;
    c.lhs_dirty[i] = 0;
    d2 = (double)d * (double)d;
    int s = i / kSlice, lane = i - s * kSlice;
    int base = c.sl_ptr[s] + lane;
    int len = c.rlen[i];
    for (int kc = 0; kc < len; kc += kGatherChunk) {
      int2 src[kGatherChunk];
      R va[kGatherChunk], vb[kGatherChunk];
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k)
        if (kc + k < len) src[k] = reinterpret_cast<const int2 *>(c.lhs_src)[base + (kc + k) * kSlice];
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k)
        if (kc + k < len) {
          va[k] = src[k].x >= 0 ? eb[src[k].x] : R(0.0);
          vb[k] = src[k].y >= 0 ? eb[src[k].y] : R(0.0);
        }
#pragma unroll
      for (int k = 0; k < kGatherChunk; ++k)
        if (kc + k < len) {
          R v = R(0.0);
          if (src[k].x >= 0) v = v + va[k];
          if (src[k].y >= 0) v = v + vb[k];
          c.offd[base + (kc + k) * kSlice] = (double)v;
        }
    }
  }
  return d2;
}

// Ends the step's LHS pass (one thread, when every block has read the flags):
// EP, NCChange and the words after the flags (see gwce.cu).
__device__ __forceinline__ void lhs_settle(const adc_ctx &c, bool rebuild, int pending, double ep) {
  int *w = (int *)(c.flags + 1);
  const int drift = !rebuild && pending;
  w[0] = rebuild;
  w[1] = 0;
  w[2] = drift;
  if (rebuild) {
    c.flags->ep = ep;
    c.flags->ncchange = 0;
    w[3] = 0;
  } else if (drift) {
    w[3] = 1;   // the drift changed every row's off-diagonals: the next rebuild gathers all
  }
  c.tickets[1] = 0;
}

// gwce.F:654-707: elevation-boundary rows and columns, OBCCoef, diagonal
// checks.  Item t < NP handles row t; item NP + q the q-th (I, J) column
// entry.
__device__ __forceinline__ void item_bc(const adc_ctx &c, double EP, int t) {
  if (t < c.np) {
    int i = t;
    if (c.is_nbd[i] >= 0) {
      c.diag[i] = EP;
      int s = i / kSlice, lane = i - s * kSlice;
      int base = c.sl_ptr[s] + lane;
      int len = c.rlen[i];
      for (int k = 0; k < len; ++k) c.offd[base + k * kSlice] = 0.0;
    }
    double d = c.diag[i];
    if (d == 0.0) {
      d = EP;
      c.diag[i] = d;
    }
    if (d < 0.0) atomicExch(&c.flags->status, ADC_ERR_DIAG);
    return;
  }
  int q = t - c.np;
  if (q >= c.n_obc) return;
  int slot = c.obc_slot[q];
  double v = 0.0;
  if (slot >= 0) {
    if (!c.obc_zero[q]) v = c.offd[slot];
    c.offd[slot] = 0.0;
  }
  c.obccoef[q] = v;
}

// ----------------------------------------------------------------- RHS
// gwce.F:1000-1617 for the 32 elements from e0, one per lane, IM=0 branches.
// `sh`: 96 values of the warp.
template <class R, bool kFast>
__device__ __forceinline__ bool warp_rhs_by(const adc_ctx &c, int e0, R *sh) {
  bool bad = false;
  const int nvalid = min(32, c.ne - e0);
  // idle lanes recompute the last element; not stored
  const int e = min(e0 + (int)(threadIdx.x & 31), c.ne - 1);
  const adc_params_t &p = c.p;
  const R DT = R(p.dt), G = R(p.g), A00 = R(p.a00), B00 = R(p.b00), C00 = R(p.c00);
  // x / DT: with a power-of-two DT, the product with its exact reciprocal
  // gives the same bits
  const bool dt2 = c.dt_pow2 != 0;
  const R IDT = R(c.inv_dt);
  const Divisor<R, kFast> by_dt(DT, IDT, bad);
  auto odt = [&](R x) { return dt2 ? x * IDT : by_dt(x, bad); };
  int n1 = c.nm[3 * e], n2 = c.nm[3 * e + 1], n3 = c.nm[3 * e + 2];
  int NCEle = c.nodecode[n1] * c.nodecode[n2] * c.nodecode[n3] * c.noff[e];
  R E0N1 = c.eta1[n1], E0N2 = c.eta1[n2], E0N3 = c.eta1[n3];
  R E1N1 = c.eta2[n1], E1N2 = c.eta2[n2], E1N3 = c.eta2[n3];
  R E1N1SQ = E1N1 * E1N1, E1N2SQ = E1N2 * E1N2, E1N3SQ = E1N3 * E1N3;
  R ESN1 = c.etas[n1], ESN2 = c.etas[n2], ESN3 = c.etas[n3];
  R U1N1 = c.uu1[n1], U1N2 = c.uu1[n2], U1N3 = c.uu1[n3];
  R V1N1 = c.vv1[n1], V1N2 = c.vv1[n2], V1N3 = c.vv1[n3];
  R QX1N1 = c.qx1[n1], QX1N2 = c.qx1[n2], QX1N3 = c.qx1[n3];
  R QY1N1 = c.qy1[n1], QY1N2 = c.qy1[n2], QY1N3 = c.qy1[n3];
  R H1N1 = c.h2[n1], H1N2 = c.h2[n2], H1N3 = c.h2[n3];
  R EVMN1 = c.evm[n1], EVMN2 = c.evm[n2], EVMN3 = c.evm[n3];
  R T0N1 = c.tau0[n1], T0N2 = c.tau0[n2], T0N3 = c.tau0[n3];
  const bool met = p.nws != 0;
  R Pr1N1 = R(0.0), Pr1N2 = R(0.0), Pr1N3 = R(0.0);
  if (met) {
    if constexpr (sizeof(R) == 4) {
      // only the gradient of PR1 is used: FP32 carries its deviation from
      // the background pressure, not the ~10 m total
      const double pb = p.prbckgrnd_mh2o;
      Pr1N1 = R(c.pr1[n1] - pb); Pr1N2 = R(c.pr1[n2] - pb); Pr1N3 = R(c.pr1[n3] - pb);
    } else {
      Pr1N1 = c.pr1[n1]; Pr1N2 = c.pr1[n2]; Pr1N3 = c.pr1[n3];
    }
  }
  const double *tk1 = c.tkm + 3 * n1, *tk2 = c.tkm + 3 * n2, *tk3 = c.tkm + 3 * n3;
  R BSXN1 = R(tk1[0]) * QX1N1 + R(tk1[2]) * QY1N1;
  R BSYN1 = R(tk1[2]) * QX1N1 + R(tk1[1]) * QY1N1;
  R BSXN2 = R(tk2[0]) * QX1N2 + R(tk2[2]) * QY1N2;
  R BSYN2 = R(tk2[2]) * QX1N2 + R(tk2[1]) * QY1N2;
  R BSXN3 = R(tk3[0]) * QX1N3 + R(tk3[2]) * QY1N3;
  R BSYN3 = R(tk3[2]) * QX1N3 + R(tk3[1]) * QY1N3;
  R AreaIE2 = c.areas[e];
  R AreaIE = AreaIE2 / R(2.0);
  R AreaIE4 = R(2.0) * AreaIE2;
  const Divisor<R, kFast> by_area(AreaIE2, bad);
  auto by_area2x = [&](R x) {   // a power of two more: the half of the quotient
    if constexpr (kFast && sizeof(R) == 8) return R(0.5) * by_area(x, bad);
    return x / AreaIE4;
  };
  R FDX1 = c.fdx[3 * e], FDX2 = c.fdx[3 * e + 1], FDX3 = c.fdx[3 * e + 2];
  R FDY1 = c.fdy[3 * e], FDY2 = c.fdy[3 * e + 1], FDY3 = c.fdy[3 * e + 2];
  R E0XGrad2A, E0YGrad2A, E1XGrad2A, E1YGrad2A, E1SQXGrad2A, E1SQYGrad2A;
  if constexpr (sizeof(R) == 4) {
    // Elevation gradients cancel metre-sized nodal values down to
    // centimetres: they are formed in FP64 and only then narrowed.
    const double *fx = c.fdx + 3 * e, *fy = c.fdy + 3 * e;
    const double a1 = c.eta1[n1], a2 = c.eta1[n2], a3 = c.eta1[n3];
    const double b1 = c.eta2[n1], b2 = c.eta2[n2], b3 = c.eta2[n3];
    E0XGrad2A = R(a1 * fx[0] + a2 * fx[1] + a3 * fx[2]);
    E0YGrad2A = R(a1 * fy[0] + a2 * fy[1] + a3 * fy[2]);
    E1XGrad2A = R(b1 * fx[0] + b2 * fx[1] + b3 * fx[2]);
    E1YGrad2A = R(b1 * fy[0] + b2 * fy[1] + b3 * fy[2]);
    E1SQXGrad2A = R(b1 * b1 * fx[0] + b2 * b2 * fx[1] + b3 * b3 * fx[2]);
    E1SQYGrad2A = R(b1 * b1 * fy[0] + b2 * b2 * fy[1] + b3 * b3 * fy[2]);
  } else {
    E0XGrad2A = E0N1 * FDX1 + E0N2 * FDX2 + E0N3 * FDX3;
    E0YGrad2A = E0N1 * FDY1 + E0N2 * FDY2 + E0N3 * FDY3;
    E1XGrad2A = E1N1 * FDX1 + E1N2 * FDX2 + E1N3 * FDX3;
    E1YGrad2A = E1N1 * FDY1 + E1N2 * FDY2 + E1N3 * FDY3;
    E1SQXGrad2A = E1N1SQ * FDX1 + E1N2SQ * FDX2 + E1N3SQ * FDX3;
    E1SQYGrad2A = E1N1SQ * FDY1 + E1N2SQ * FDY2 + E1N3SQ * FDY3;
  }
  R Tau0XGrad2A = T0N1 * FDX1 + T0N2 * FDX2 + T0N3 * FDX3;
  R Tau0YGrad2A = T0N1 * FDY1 + T0N2 * FDY2 + T0N3 * FDY3;
  R EVMXGrad = by_area(EVMN1 * FDX1 + EVMN2 * FDX2 + EVMN3 * FDX3, bad);
  R EVMYGrad = by_area(EVMN1 * FDY1 + EVMN2 * FDY2 + EVMN3 * FDY3, bad);
  R EVMAvgODT = odt(div3(EVMN1 + EVMN2 + EVMN3));
  R MX = by_area(EVMXGrad * (QX1N1 * FDX1 + QX1N2 * FDX2 + QX1N3 * FDX3) +
               EVMYGrad * (QY1N1 * FDX1 + QY1N2 * FDX2 + QY1N3 * FDX3) -
               EVMAvgODT * (ESN1 * FDX1 + ESN2 * FDX2 + ESN3 * FDX3), bad);
  R MY = by_area(EVMXGrad * (QX1N1 * FDY1 + QX1N2 * FDY2 + QX1N3 * FDY3) +
               EVMYGrad * (QY1N1 * FDY1 + QY1N2 * FDY2 + QY1N3 * FDY3) -
               EVMAvgODT * (ESN1 * FDY1 + ESN2 * FDY2 + ESN3 * FDY3), bad);
  R CorifAvg = div3(c.corif[n1] + c.corif[n2] + c.corif[n3]);
  R Tau0Avg = div3(T0N1 + T0N2 + T0N3);
  R Tau0QXAvg = div3(T0N1 * QX1N1 + T0N2 * QX1N2 + T0N3 * QX1N3);
  R Tau0QYAvg = div3(T0N1 * QY1N1 + T0N2 * QY1N2 + T0N3 * QY1N3);
  R U1Avg = div3(U1N1 + U1N2 + U1N3);
  R V1Avg = div3(V1N1 + V1N2 + V1N3);
  R QX1Avg = div3(QX1N1 + QX1N2 + QX1N3);
  R QY1Avg = div3(QY1N1 + QY1N2 + QY1N3);
  R ESAvg = div3(ESN1 + ESN2 + ESN3);
  R DPAvg = div3(c.dp[n1] + c.dp[n2] + c.dp[n3]);
  R al = c.alphal[e];
  R GDPAvgOAreaIE4 = by_area2x(al * G * DPAvg);
  R GDPAvgOAreaIE4_S0 = GDPAvgOAreaIE4;   // DPAvgS0 == DPAvg when IFNL_HDP = 0
  R HAvg = div3(H1N1 + H1N2 + H1N3);
  R GHAvg = al * G * HAvg;
  R GHAvgOAreaIE2 = by_area(GHAvg, bad);
  R BSXAvg = div3(BSXN1 + BSXN2 + BSXN3);
  R BSYAvg = div3(BSYN1 + BSYN2 + BSYN3);
  R WSXAvg = R(0.0), WSYAvg = R(0.0);
  if (met) {
    WSXAvg = div3(c.wsx1[n1] + c.wsx1[n2] + c.wsx1[n3]);
    WSYAvg = div3(c.wsy1[n1] + c.wsy1[n2] + c.wsy1[n3]);
  }
  R MsFacR = div12(odt(AreaIE * ((dt2 ? IDT : R(1.0) / DT) - Tau0Avg / R(2.0))));
  R GOAreaIE4 = by_area2x(al * G);
  R Tau0SpaVar = div6(QX1Avg * Tau0XGrad2A + QY1Avg * Tau0YGrad2A);
  R A00pB00 = A00 + B00;
  R fa = p.ifnlfa * GOAreaIE4;
  R JXAvg = CorifAvg * QY1Avg - fa * E1SQXGrad2A -
                 GHAvgOAreaIE2 * (Pr1N1 * FDX1 + Pr1N2 * FDX2 + Pr1N3 * FDX3) + WSXAvg -
                 BSXAvg + MX + Tau0QXAvg;
  R JYAvg = -CorifAvg * QX1Avg - fa * E1SQYGrad2A -
                 GHAvgOAreaIE2 * (Pr1N1 * FDY1 + Pr1N2 * FDY2 + Pr1N3 * FDY3) + WSYAvg -
                 BSYAvg + MY + Tau0QYAvg;
  JXAvg = JXAvg - by_area(p.ifnlct * (QX1Avg * (U1N1 * FDX1 + U1N2 * FDX2 + U1N3 * FDX3) +
                              QY1Avg * (U1N1 * FDY1 + U1N2 * FDY2 + U1N3 * FDY3)), bad) +
          odt(p.ifnlcat * U1Avg * ESAvg);
  JYAvg = JYAvg - by_area(p.ifnlct * (QX1Avg * (V1N1 * FDX1 + V1N2 * FDX2 + V1N3 * FDX3) +
                              QY1Avg * (V1N1 * FDY1 + V1N2 * FDY2 + V1N3 * FDY3)), bad) +
          odt(p.ifnlcat * V1Avg * ESAvg);
  R c0 = GDPAvgOAreaIE4_S0, c1 = GDPAvgOAreaIE4;
  R T1 = (2 * ESN1 + 1 * (ESN2 + ESN3)) * MsFacR -
              c0 * (C00 * (FDX1 * E0XGrad2A + FDY1 * E0YGrad2A)) -
              c1 * (A00pB00 * (FDX1 * E1XGrad2A + FDY1 * E1YGrad2A)) +
              (JXAvg * FDX1 + JYAvg * FDY1) * R(0.5) + Tau0SpaVar;
  R T2 = (2 * ESN2 + 1 * (ESN1 + ESN3)) * MsFacR -
              c0 * (C00 * (FDX2 * E0XGrad2A + FDY2 * E0YGrad2A)) -
              c1 * (A00pB00 * (FDX2 * E1XGrad2A + FDY2 * E1YGrad2A)) +
              (JXAvg * FDX2 + JYAvg * FDY2) * R(0.5) + Tau0SpaVar;
  R T3 = (2 * ESN3 + 1 * (ESN1 + ESN2)) * MsFacR -
              c0 * (C00 * (FDX3 * E0XGrad2A + FDY3 * E0YGrad2A)) -
              c1 * (A00pB00 * (FDX3 * E1XGrad2A + FDY3 * E1YGrad2A)) +
              (JXAvg * FDX3 + JYAvg * FDY3) * R(0.5) + Tau0SpaVar;
  R nc = (R)NCEle;
  const R o[3] = {T1 * nc, T2 * nc, T3 * nc};
  warp_store_k<3>(reinterpret_cast<R *>(c.ebuf) + 3 * (size_t)e0, o, nvalid, sh);
  return bad;
}

template <class R>
__device__ __forceinline__ void warp_rhs(const adc_ctx &c, int e0, R *sh) {
  if constexpr (sizeof(R) == 8) {
    if (!__any_sync(0xffffffffu, warp_rhs_by<R, true>(c, e0, sh))) return;
  }
  warp_rhs_by<R, false>(c, e0, sh);
}

// GWCE_LV gather (element order) fused with gwce.F:1622-1631.
template <class R>
__device__ __forceinline__ void node_rhs(const adc_ctx &c, int i) {
  const R *eb = reinterpret_cast<const R *>(c.ebuf);
  R v = R(0.0);
  const int q0 = c.n2e_ptr[i], q1 = c.n2e_ptr[i + 1];
  for (int qc = q0; qc < q1; qc += kGatherChunk) {
    int ek[kGatherChunk];
    R x[kGatherChunk];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) ek[k] = c.n2e[qc + k];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) x[k] = eb[ek[k]];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) v = v + x[k];
  }
  c.gwce_lv[i] = (double)v;
  c.eta1[i] = c.eta2[i];
  c.h1[i] = c.h2[i];
  c.eta2[i] = 0.0;
}

// gwce.F:1638-1651 periodic elevation BC and :1846-1850 load-vector rows.
__device__ __forceinline__ void bnd_eta(const adc_ctx &c, const adc_step_t &st, double EP, int I) {
  int b = c.nbd[I];
  double e2 = 0.0;   // ETA2 was zeroed in node_rhs
  for (int J = 0; J < c.nbfr; ++J) {
    int NCYC = 0;
    if (c.per[J] != 0.0) NCYC = (int)(st.timeh / c.per[J]);
    double ARGJ = c.amig[J] * (st.timeh - NCYC * c.per[J]) + c.face[J];
    double RFF = c.ff[J] * st.rampelev;
    double ARG = ARGJ - c.efa[J + (size_t)c.nbfr * I];
    e2 = e2 + c.emo[J + (size_t)c.nbfr * I] * RFF * cos(ARG);
  }
  if (c.eser_on) {   // non-periodic elevations, gwce.F:1668-1673
    const SeriesState &ss = c.sstate[0];
    const size_t r1 = (size_t)ss.k * c.neta, r2 = r1 + c.neta;
    e2 = e2 + st.rampelev * (c.eser[r1 + I] + ss.ratio * (c.eser[r2 + I] - c.eser[r1 + I]));
  }
  c.eta2[b] = e2;
  double es = e2 - c.eta1[b];
  c.etas[b] = es;
  c.gwce_lv[b] = es * c.nodecode[b] * EP;
}

// gwce.F:1851-1854 column correction, per affected neighbour in (I, J) order.
__device__ __forceinline__ void bnd_obc(const adc_ctx &c, int r) {
  int nb = c.obc_rhs_node[r];
  double v = c.gwce_lv[nb];
  for (int q = c.obc_rhs_ptr[r]; q < c.obc_rhs_ptr[r + 1]; ++q)
    v = v - c.etas[c.obc_rhs_b[q]] * c.obccoef[c.obc_rhs_ent[q]];
  c.gwce_lv[nb] = v;
}

// -------------------------------------------------------------- wet/dry
// D1, wetdry.F:234-285.
__device__ __forceinline__ void node_d1(const adc_ctx &c, int i) {
  double eta = c.eta2[i];
  if (d1_dries(c.nodecode[i], c.dp[i], c.p.h0, eta)) {
    c.eta2[i] = eta;
    c.nnodecode[i] = 0;
    c.nodecode[i] = 0;
    atomicAdd(&c.flags->ncchange, 1);
  }
}

// -------------------------------------------------------- flux boundaries
// One thread: per active series, the record pair and ratio of this step.
// The reference reads the next record when TimeLoc passes the later record
// time, at most once per step (gwce.F:1660-1668, timestep.F:882-900).
__device__ inline void one_series(const adc_ctx &c, double timeloc) {
  for (int s = 0; s < 2; ++s) {
    if (!(s == 0 ? c.eser_on : c.fser_on)) continue;
    SeriesState &st = c.sstate[s];
    const int nrec = s == 0 ? c.eser_nrec : c.fser_nrec;
    const double inc = s == 0 ? c.eser_interval : c.fser_interval;
    if (timeloc > st.t2) {
      st.t1 = st.t2;
      st.t2 = st.t1 + inc;
      st.k = st.k + 1;
      if (st.k + 1 >= nrec) {   // the file has no further record
        st.err = 1;
        c.flags->status = ADC_ERR_ARG;
        st.k = nrec - 2;
      }
    }
    st.ratio = (timeloc - st.t1) / inc;
  }
}

// COMPUTE_INTERNAL_BOUNDARY_FLUX (weir_boundary.F90:1775-1942, the default
// wet-edge formulation without averaging); the square roots stand for the
// reference's **0.5.
__device__ inline double internal_barrier_flux(const adc_ctx &c, int I, double ramp) {
  const int n1 = c.bnv[I], n2 = c.ibconn[I], kind = c.ibkind[I];
  const int *nc = c.nodecode;
  int wn1 = 0, wn2 = 0;   // wet neighbours along the barrier on each side
  if (kind == 0) {
    wn1 = wn1 + nc[c.bnv[I + 1]];
    wn2 = wn2 + nc[c.ibconn[I + 1]];
  } else if (kind == 1) {
    wn1 = wn1 + nc[c.bnv[I - 1]];
    wn2 = wn2 + nc[c.ibconn[I - 1]];
  } else {
    wn1 = wn1 + nc[c.bnv[I - 1]];
    wn1 = wn1 + nc[c.bnv[I + 1]];
    wn2 = wn2 + nc[c.ibconn[I + 1]];
    wn2 = wn2 + nc[c.ibconn[I - 1]];
  }
  const double R1 = c.eta2[n1] - c.binht[I], R2 = c.eta2[n2] - c.binht[I];
  const double R1F = 2.0 * R1 / 3.0, R2F = 2.0 * R2 / 3.0;
  const double G = c.p.g, BARMIN = 0.04;
  double flux = 0.0;
  if ((R1 < 0.0) && (R2 < 0.0)) {
    flux = 0.0;
  } else if (fabs(R1 - R2) < 0.01) {
    flux = 0.0;
  } else if ((R1 > R2) && (R1 > BARMIN)) {   // this side is the source
    if (nc[n1] == 0 || wn1 == 0) flux = 0.0;
    else if (R2 > R1F) flux = -ramp * R2 * c.bincfsb[I] * sqrt(2.0 * G * (R1 - R2));
    else flux = -ramp * c.bincfsp[I] * R1F * sqrt(R1F * G);
  } else if ((R2 > R1) && (R2 > BARMIN)) {   // this side receives
    if (nc[n2] == 0 || wn2 == 0) {
      flux = 0.0;
    } else {
      if (R1 > R2F) flux = ramp * R1 * c.bincfsb[I] * sqrt(2.0 * G * (R2 - R1));
      else flux = ramp * c.bincfsp[I] * R2F * sqrt(R2F * G);
      c.nib[n1] = 1;
    }
  }
  return flux;
}

// COMPUTE_CROSS_BARRIER_PIPE_FLUX (weir_boundary.F90:2469-2579); the
// reference's **0.5 as square roots and PIPEDIAM**2 as a product.
__device__ inline double pipe_flux(const adc_ctx &c, int I, double ramp) {
  const int n1 = c.bnv[I], n2 = c.ibconn[I];
  const double *pp = c.pipe;
  const double ht = pp[I], coef = pp[c.nvel + I], diam = pp[2 * c.nvel + I];
  const double G = c.p.g, BARMIN = 0.04, PI = 3.141592653589793;
  const double R1 = c.eta2[n1] - ht, R2 = c.eta2[n2] - ht;
  if ((R1 < 0.0) && (R2 < 0.0)) return 0.0;
  if (fabs(R1 - R2) < BARMIN) return 0.0;
  double flux = 0.0;
  if ((R1 > R2) && (R1 > BARMIN)) {   // outward
    if (R2 <= 0.0) {
      flux = c.nodecode[n1] == 0 ? 0.0
                                 : -ramp * 0.25 * PI * (diam * diam) * sqrt(2.0 * G * R1 / (1.0 + coef));
    } else {
      return c.nodecode[n1] == 0 ? 0.0
                                 : -ramp * 0.25 * PI * (diam * diam) * sqrt(2.0 * G * (R1 - R2) / coef);
    }
  }
  if ((R2 > R1) && (R2 > BARMIN)) {   // inward
    if (c.nodecode[n2] == 0) return 0.0;
    if (R1 <= 0.0) flux = ramp * 0.25 * PI * (diam * diam) * sqrt(2.0 * G * R2 / (1.0 + coef));
    else flux = ramp * 0.25 * PI * (diam * diam) * sqrt(2.0 * G * (R2 - R1) / coef);
    c.nib[n1] = 1;
  }
  return flux;
}


// The discharge (and elevation) of boundary entry I this step.
__device__ inline void bnd_forcing(const adc_ctx &c, const adc_step_t &st, int I) {
  double *qn0 = c.qn, *qn1 = c.qn + c.nvel, *qn2 = c.qn + 2 * c.nvel;
  double *en0 = c.en, *en1 = c.en + c.nvel, *en2 = c.en + 2 * c.nvel;
  qn0[I] = qn1[I];
  qn1[I] = qn2[I];
  en0[I] = en1[I];
  en1[I] = en2[I];
  double q = 0.0, el = 0.0;
  const int lb = c.blbc[I];
  if (c.flux_on && (lb == 2 || lb == 12 || lb == 22 || lb == 32 || lb == 52)) {
    const int nf = c.nffr;
    const size_t nfv = (size_t)nf * c.nvel;
    const double *famig = c.fconst, *fper = famig + nf, *fff = fper + nf, *fface = fff + nf;
    const double *qnam = c.fqn, *qnph = c.fqn + nfv, *enam = qnph + nfv, *enph = enam + nfv;
    const bool coupled = lb == 32 && c.fen;
    for (int J = 0; J < nf; ++J) {
      int NCYC = 0;
      if (fper[J] != 0.0) NCYC = (int)(st.timeh / fper[J]);
      const double ARGJ = famig[J] * (st.timeh - NCYC * fper[J]) + fface[J];
      const double RFF = fff[J] * st.rampextflux;
      q = q + qnam[J + (size_t)nf * I] * RFF * cos(ARGJ - qnph[J + (size_t)nf * I]);
      if (coupled) el = el + enam[J + (size_t)nf * I] * RFF * cos(ARGJ - enph[J + (size_t)nf * I]);
    }
  } else if (c.fser_on) {   // timestep.F:900-902, every entry
    const SeriesState &ss = c.sstate[1];
    const size_t r1 = (size_t)ss.k * c.nvel, r2 = r1 + c.nvel;
    q = st.rampextflux * (c.fser_q[r1 + I] + ss.ratio * (c.fser_q[r2 + I] - c.fser_q[r1 + I]));
    el = st.rampextflux * (c.fser_e[r1 + I] + ss.ratio * (c.fser_e[r2 + I] - c.fser_e[r1 + I]));
  }
  if (lb == 3 || lb == 13 || lb == 23) {
    // the weir formula with g and BARMIN = 0.04 m (weir_boundary.F90:51);
    // (RBARWL g)^0.5 as a square root
    const double RBARWL = 2.0 * (c.eta2[c.bnv[I]] - c.barht[I]) / 3.0;
    q = RBARWL > 0.04 ? -st.rampintflux * c.barcf[I] * RBARWL * sqrt(RBARWL * c.p.g) : 0.0;
  }
  if (lb == 4 || lb == 24 || lb == 5 || lb == 25) q = internal_barrier_flux(c, I, st.rampintflux);
  if (lb == 5 || lb == 25) q = q + pipe_flux(c, I, st.rampintflux);   // timestep.F:1034-1044
  qn2[I] = q;
  en2[I] = el;
  if (lb == 52) {
    const int n = c.bnv[I];
    if (st.it == c.flux_settling_it) {
      c.etadisc_b[I] = c.eta2[n];
      c.elevdisc[I] = c.eta2[n];
    } else if (!c.flags->etadisc_done && st.it > c.flux_settling_it) {
      c.elevdisc[I] = c.etadisc_b[I];
    }
  }
  if (lb == 30 || lb == 40 || lb == 41) {
    const int n = c.bnv[I];
    const double UN1 = c.uu1[n] * c.bcsii[I] + c.vv1[n] * c.bsiii[I];
    qn1[I] = c.h2[n] * UN1;
  }
}

// The force of each boundary entry (gwce.F:1783-1815): LBCODEI <= 29 from
// the specified flux, 30 the radiation condition with the saved H1, 52 the
// specified flux plus, after FluxSettlingIT, the radiation term.
__device__ inline void bnd_qforce(const adc_ctx &c, int it, int J) {
  const double *qn0 = c.qn, *qn1 = c.qn + c.nvel, *qn2 = c.qn + 2 * c.nvel;
  const int n = c.bnv[J];
  if (c.blbc[J] == 32) {   // gwce.F:1792-1797
    const double *en0 = c.en, *en1 = c.en + c.nvel, *en2 = c.en + 2 * c.nvel;
    const double CELERITY = sqrt(c.p.g * c.h1[n]);
    const double DT2 = c.p.dt * 2.0;
    c.qforce[J] = (qn2[J] - qn0[J]) / DT2 - CELERITY * (2.0 * c.etas[n] - (en2[J] - en0[J])) / DT2 +
                  c.tau0[n] * (qn1[J] - CELERITY * (c.eta1[n] - en1[J]));
    return;
  }
  if (c.blbc[J] == 40 || c.blbc[J] == 41) {   // gwce.F:1804-1805
    c.qforce[J] = -(qn1[J] - qn0[J]) / c.p.dt - c.tau0[n] * (qn1[J] + qn0[J]) / 2.0;
    return;
  }
  if (c.blbc[J] == 30) {
    const double CELERITY = sqrt(c.p.g * c.h1[n]);
    c.qforce[J] = -CELERITY * c.etas[n] / c.p.dt - c.tau0[n] * qn1[J];
    return;
  }
  const double DT2 = c.p.dt * 2.0;
  double q = (qn2[J] - qn0[J]) / DT2 + c.tau0[n] * qn1[J];
  if (c.blbc[J] == 52 && it > c.flux_settling_it) {
    const double Celerity = sqrt(c.p.g * c.h1[n]);
    q = q - Celerity * (c.etas[n] / c.p.dt + c.tau0[n] * (c.eta1[n] - c.elevdisc[J]));
  }
  c.qforce[J] = q;
}

// Boundary node k of the line integral: its contributions in entry order.
__device__ inline void bnd_flux_rhs(const adc_ctx &c, int k) {
  const int n = c.fx_node[k];
  double v = c.gwce_lv[n];
  for (int q = c.fx_ptr[k]; q < c.fx_ptr[k + 1]; ++q) {
    const int ent = c.fx_ent[q], j = ent >> 1;
    const int NCI = c.nodecode[c.bnv[j - 1]], NCJ = c.nodecode[c.bnv[j]];
    const double B = NCI * NCJ * c.bbl[j - 1] / 4.0;
    const double qi = c.qforce[j - 1], qj = c.qforce[j];
    if ((ent & 1) == 0) v = v + B * (2.0 * qi + qj);   // the segment's first node
    else v = v + B * (2.0 * qj + qi);                  // its second node
  }
  c.gwce_lv[n] = v;
}

__device__ __forceinline__ double hyb_term(const adc_params_t &p, double h1) {
  if (p.ifhybf == 0) return 0.0;
  return p.ifhybf * pow(1.0 + pow(p.hbreak / h1, p.ftheta), p.fgamma / p.ftheta);
}


constexpr int kW1Block = 256;
constexpr int kChainFast = 1024;   // W1 events resolved in shared memory at a time

// W1, wetdry.F:332-809, plus NOFFOLD/NOFF initialisation (:222-225), for the
// vb-th block of 256 elements.
__device__ __forceinline__ void block_w1(const adc_ctx &c, int vb) {
  const int t = (int)threadIdx.x;
  const int e = vb * kW1Block + t;
  bool ev = false;
  int ea = 0, eb = 0;
  double ec = 0.0;
  if (e < c.ne) {
    c.noffold[e] = c.noff[e];
    c.noff[e] = 1;
    int NM1 = c.nm[3 * e], NM2 = c.nm[3 * e + 1], NM3 = c.nm[3 * e + 2];
    int nc1 = c.nodecode[NM1], nc2 = c.nodecode[NM2], nc3 = c.nodecode[NM3];
    if (nc1 + nc2 + nc3 == 2) {
      const adc_params_t &p = c.p;
      const double HOFF = 1.2 * p.h0;
      double HT1 = c.dp[NM1] + c.eta2[NM1];
      double HT2 = c.dp[NM2] + c.eta2[NM2];
      double HT3 = c.dp[NM3] + c.eta2[NM3];
      int wa = -1, wb = 0, dry = 0;
      double ha = 0, hb = 0;
      if (nc1 == 1 && nc2 == 1) { wa = NM1; wb = NM2; dry = NM3; ha = HT1; hb = HT2; }
      else if (nc2 == 1 && nc3 == 1) { wa = NM2; wb = NM3; dry = NM1; ha = HT2; hb = HT3; }
      else if (nc3 == 1 && nc1 == 1) { wa = NM3; wb = NM1; dry = NM2; ha = HT3; hb = HT1; }
      if (wa >= 0 && ha >= HOFF && hb >= HOFF) {
        int nm123 = wa;
        if (c.eta2[wb] > c.eta2[wa]) nm123 = wb;
        double dy = c.y[dry] - c.y[nm123], dx = c.x[dry] - c.x[nm123];
        double deldist = sqrt(dy * dy + dx * dx);
        double deleta = c.eta2[nm123] - c.eta2[dry];
        if (deleta < 0.0) deleta = 0.0;
        double h1 = c.eta2[nm123] + c.dp[nm123];
        double fr = c.fric[nm123];
        double tkw = fr * (p.iflinbf + (p.velmin / h1) * (p.ifnlbf + hyb_term(p, h1)));
        double tkwet = (tkw < 0.0001) ? 0.0001 : tkw;   // MAX(., 0.0001)
        double vel = p.g * (deleta / deldist) / tkwet;
        if (vel > p.velmin) {
          c.nnodecode[dry] = 1;
          double tv = fr * (p.iflinbf + (1.0 * vel / h1) * (p.ifnlbf + hyb_term(p, h1)));
          double cap = 2.0 / p.dt;
          ec = (tv < cap) ? tv : cap;
          ea = nm123;
          eb = (nm123 == wa) ? wb : wa;
          ev = true;
        }
      }
    }
  }
  // block-local ordered compaction of the events
  __shared__ int wcnt[kW1Block / 32];
  unsigned m = __ballot_sync(0xffffffffu, ev);
  const int lane = t & 31, w = t >> 5;
  if (lane == 0) wcnt[w] = __popc(m);
  __syncthreads();
  int off = 0, tot = 0;
  for (int k = 0; k < kW1Block / 32; ++k) {
    if (k < w) off += wcnt[k];
    tot += wcnt[k];
  }
  // each event goes to its block's ordered slot and, while the step has at
  // most kChainFast events, to an unordered list tagged with its element
  __shared__ int s_ubase;
  if (t == 0) {
    c.ev_cnt[vb] = tot;
    s_ubase = tot ? atomicAdd(&c.flags->n_w1_events, tot) : 0;
  }
  __syncthreads();
  if (ev) {
    const int r = off + __popc(m & ((1u << lane) - 1u));
    const int pos = vb * kW1Block + r;
    c.ev_a[pos] = ea;
    c.ev_b[pos] = eb;
    c.ev_c[pos] = ec;
    const int u = s_ubase + r;
    if (u < kChainFast) {
      c.evu_i[3 * u] = ea;
      c.evu_i[3 * u + 1] = eb;
      c.evu_i[3 * u + 2] = e;
      c.evu_c[u] = ec;
    }
  }
}

// W2a/W2b with internal barriers: NIBCNT(i) sums NIBNODECODE over the nodes
// of every element around node i (wetdry.F:813-816, an integer sum, so its
// element order does not matter), and a node with NIBCNT > 0 is wet
// (:1086-1090).
__device__ __forceinline__ void node_w2b(const adc_ctx &c, int i) {
  int cnt = 0;
  for (int q = c.n2e_ptr[i]; q < c.n2e_ptr[i + 1]; ++q) {
    const int e = c.n2e[q] / 3;
    cnt += c.nib[c.nm[3 * e]] + c.nib[c.nm[3 * e + 1]] + c.nib[c.nm[3 * e + 2]];
  }
  c.nibcnt[i] = cnt;
  if (cnt > 0 && c.nnodecode[i] == 0) c.nnodecode[i] = 1;
}

// DE1 (wetdry.F:1110-1162), then NCEle for D2 and the NOFF change count
// (:1428-1430).
__device__ __forceinline__ void elem_de1(const adc_ctx &c, int e) {
  int NM1 = c.nm[3 * e], NM2 = c.nm[3 * e + 1], NM3 = c.nm[3 * e + 2];
  const double HOFF = 1.2 * c.p.h0;
  double E1 = c.eta2[NM1], E2 = c.eta2[NM2], E3 = c.eta2[NM3];
  double H1 = c.dp[NM1] + E1, H2 = c.dp[NM2] + E2, H3 = c.dp[NM3] + E3;
  int noff = c.noff[e];
  // elements with a barrier-receiving node at every vertex keep NOFF (:1114)
  const bool receiving = c.nfluxib && c.nibcnt[NM1] * c.nibcnt[NM2] * c.nibcnt[NM3] != 0;
  if (!receiving) {
    if ((E1 >= E2) && (E2 > E3)) if ((H1 < HOFF) || (H2 < HOFF)) noff = 0;
    if ((E2 >= E3) && (E3 > E1)) if ((H2 < HOFF) || (H3 < HOFF)) noff = 0;
    if ((E3 >= E1) && (E1 > E2)) if ((H3 < HOFF) || (H1 < HOFF)) noff = 0;
    if ((E1 >= E3) && (E3 > E2)) if ((H1 < HOFF) || (H3 < HOFF)) noff = 0;
    if ((E2 >= E1) && (E1 > E3)) if ((H2 < HOFF) || (H1 < HOFF)) noff = 0;
    if ((E3 >= E2) && (E2 > E1)) if ((H3 < HOFF) || (H2 < HOFF)) noff = 0;
  }
  c.noff[e] = noff;
  c.ncele[e] = c.nnodecode[NM1] * c.nnodecode[NM2] * c.nnodecode[NM3] * noff;
  if (noff != c.noffold[e]) atomicAdd(&c.flags->ncchange, 1);
}

// D2 (wetdry.F:1361-1391), NODECODE update (:1413-1418) and the H2 update
// of timestep.F:1097-1099.
__device__ __forceinline__ void node_d2(const adc_ctx &c, int i) {
  int mju = 0;
  double ta = 0.0;
  const int q0 = c.n2e_ptr[i], q1 = c.n2e_ptr[i + 1];
  for (int qc = q0; qc < q1; qc += kGatherChunk) {
    int ee[kGatherChunk], nc[kGatherChunk];
    double ar[kGatherChunk];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) ee[k] = c.n2e[qc + k] / 3;
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (qc + k < q1) {
        nc[k] = c.ncele[ee[k]];
        ar[k] = c.areas[ee[k]];
      }
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (qc + k < q1) {
        mju += nc[k];
        ta = ta + nc[k] * ar[k] / 2.0;
      }
  }
  c.totalarea[i] = ta;
  int nn = c.nnodecode[i];
  if (nn == 1 && mju == 0) {
    nn = 0;
    c.nnodecode[i] = 0;
  }
  c.mju[i] = (mju == 0) ? 1 : mju;
  if (nn != c.nodecode[i]) {
    c.nodecode[i] = nn;
    atomicAdd(&c.flags->ncchange, 1);
  }
  c.h2[i] = c.dp[i] + c.p.ifnlfa * c.eta2[i];
}

// computeAlpha, wetdry.F:1561-1652: ALPHAL of one element.
__device__ __forceinline__ double elem_alpha(const adc_ctx &c, int e) {
  int NM1 = c.nm[3 * e], NM2 = c.nm[3 * e + 1], NM3 = c.nm[3 * e + 2];
  double al = 1.0;
  int NCEle = c.nodecode[NM1] * c.nodecode[NM2] * c.nodecode[NM3] * c.noff[e];
  if (NCEle == 1) {
    double E1 = c.eta2[NM1], E2 = c.eta2[NM2], E3 = c.eta2[NM3];
    double HN1 = E1 + c.dp[NM1], HN2 = E2 + c.dp[NM2], HN3 = E3 + c.dp[NM3];
    if ((HN1 <= 5.0e-1) || (HN2 <= 5.0e-1) || (HN3 <= 5.0e-1)) {
      double FDX1 = c.fdx[3 * e], FDX2 = c.fdx[3 * e + 1], FDX3 = c.fdx[3 * e + 2];
      double FDY1 = c.fdy[3 * e], FDY2 = c.fdy[3 * e + 1], FDY3 = c.fdy[3 * e + 2];
      double D1 = c.dp[NM1], D2 = c.dp[NM2], D3 = c.dp[NM3];
      double DPDXA = D1 * FDX1 + D2 * FDX2 + D3 * FDX3;
      double DPDYA = D1 * FDY1 + D2 * FDY2 + D3 * FDY3;
      double DETADXA = E1 * FDX1 + E2 * FDX2 + E3 * FDX3;
      double DETADYA = E1 * FDY1 + E2 * FDY2 + E3 * FDY3;
      double ar = c.areas[e];
      double DPM = sqrt(DPDXA * DPDXA + DPDYA * DPDYA) / ar;
      if (DPM > 1.0e-5) {
        double DDTMP = DETADXA * (-DPDXA) + DETADYA * (-DPDYA);
        if (fabs(DDTMP) > 1.0e-12)
          al = c.p.slim * (sqrt(DPDXA * DPDXA + DPDYA * DPDYA) / ((1.0 / ar) * (DDTMP)));
        else
          al = 1.0;
      } else {
        double DETAM = sqrt(DETADXA * DETADXA + DETADYA * DETADYA) / ar;
        if (fabs(DETAM) > 1.0e-12) al = c.p.slim / DETAM;
        else al = 1.0;
      }
      if (al <= 0.0) al = 1.0;
      if (al >= 1.0) al = 1.0;
    }
  }
  return al;
}

// ------------------------------------------------------------- momentum
// Element terms (momentum.F:298-699) for the 32 elements from e0, one per
// lane.  `sh`: 192 values of the warp.  `alpha`: ALPHAL is formed here
// (computeAlpha ends the wet/dry step that precedes).
template <class R, bool kFast>
__device__ __forceinline__ bool warp_mom_by(const adc_ctx &c, int e0, R *sh, bool alpha) {
  bool bad = false;
  const int nvalid = min(32, c.ne - e0);
  const int e = min(e0 + (int)(threadIdx.x & 31), c.ne - 1);   // idle lanes are not stored
  const adc_params_t &p = c.p;
  const R DT = R(p.dt);
  const R THIRD = R(R(1.0)) / R(R(3.0)), GO2 = R(p.g) / R(R(2.0));
  const bool met = p.nws != 0;
  int n1 = c.nm[3 * e], n2 = c.nm[3 * e + 1], n3 = c.nm[3 * e + 2];
  int NCEle = c.nodecode[n1] * c.nodecode[n2] * c.nodecode[n3] * c.noff[e];
  R U1N1 = c.uu1[n1], U1N2 = c.uu1[n2], U1N3 = c.uu1[n3];
  R V1N1 = c.vv1[n1], V1N2 = c.vv1[n2], V1N3 = c.vv1[n3];
  R H1N1 = c.h1[n1], H1N2 = c.h1[n2], H1N3 = c.h1[n3];
  R AreaIE2 = c.areas[e];
  R AreaIE = R(0.5) * AreaIE2;
  R FDX1 = c.fdx[3 * e], FDX2 = c.fdx[3 * e + 1], FDX3 = c.fdx[3 * e + 2];
  R FDY1 = c.fdy[3 * e], FDY2 = c.fdy[3 * e + 1], FDY3 = c.fdy[3 * e + 2];
  R U1Avg = THIRD * (U1N1 + U1N2 + U1N3);
  R V1Avg = THIRD * (V1N1 + V1N2 + V1N3);
  R DU1DXA = (U1N1 * FDX1 + U1N2 * FDX2 + U1N3 * FDX3) * R(0.5);
  R DU1DYA = (U1N1 * FDY1 + U1N2 * FDY2 + U1N3 * FDY3) * R(0.5);
  R DV1DXA = (V1N1 * FDX1 + V1N2 * FDX2 + V1N3 * FDX3) * R(0.5);
  R DV1DYA = (V1N1 * FDY1 + V1N2 * FDY2 + V1N3 * FDY3) * R(0.5);
  R EVMEle = THIRD * (c.evm[n1] + c.evm[n2] + c.evm[n3]);
  double ald;
  if (alpha) {
    ald = elem_alpha(c, e);
    if ((int)(threadIdx.x & 31) < nvalid) c.alphal[e] = ald;
  } else {
    ald = c.alphal[e];
  }
  R al = ald;
  R B11 = al * c.eta1[n1], B21 = al * c.eta2[n1];
  R B12 = al * c.eta1[n2], B22 = al * c.eta2[n2];
  R B13 = al * c.eta1[n3], B23 = al * c.eta2[n3];
  if (met) {
    if constexpr (sizeof(R) == 4) {
      // only gradients of B are used: FP32 carries the pressure's deviation
      // from the background, not the ~10 m total
      const double pb = p.prbckgrnd_mh2o;
      B11 = B11 + R(c.pr1[n1] - pb); B21 = B21 + R(c.pr2[n1] - pb);
      B12 = B12 + R(c.pr1[n2] - pb); B22 = B22 + R(c.pr2[n2] - pb);
      B13 = B13 + R(c.pr1[n3] - pb); B23 = B23 + R(c.pr2[n3] - pb);
    } else {
      B11 = B11 + c.pr1[n1]; B21 = B21 + c.pr2[n1];
      B12 = B12 + c.pr1[n2]; B22 = B22 + c.pr2[n2];
      B13 = B13 + c.pr1[n3]; B23 = B23 + c.pr2[n3];
    }
  }
  R DBTPDX1A, DBTPDX2A, DBTPDY1A, DBTPDY2A;
  if constexpr (sizeof(R) == 4) {
    // barotropic-pressure gradients cancel metre-sized nodal values: FP64,
    // then narrowed
    const double *fx = c.fdx + 3 * e, *fy = c.fdy + 3 * e;
    double b11 = ald * c.eta1[n1], b21 = ald * c.eta2[n1];
    double b12 = ald * c.eta1[n2], b22 = ald * c.eta2[n2];
    double b13 = ald * c.eta1[n3], b23 = ald * c.eta2[n3];
    if (met) {
      b11 += c.pr1[n1]; b21 += c.pr2[n1];
      b12 += c.pr1[n2]; b22 += c.pr2[n2];
      b13 += c.pr1[n3]; b23 += c.pr2[n3];
    }
    DBTPDX1A = R(b11 * fx[0] + b12 * fx[1] + b13 * fx[2]);
    DBTPDX2A = R(b21 * fx[0] + b22 * fx[1] + b23 * fx[2]);
    DBTPDY1A = R(b11 * fy[0] + b12 * fy[1] + b13 * fy[2]);
    DBTPDY2A = R(b21 * fy[0] + b22 * fy[1] + b23 * fy[2]);
  } else {
    DBTPDX1A = B11 * FDX1 + B12 * FDX2 + B13 * FDX3;
    DBTPDX2A = B21 * FDX1 + B22 * FDX2 + B23 * FDX3;
    DBTPDY1A = B11 * FDY1 + B12 * FDY2 + B13 * FDY3;
    DBTPDY2A = B21 * FDY1 + B22 * FDY2 + B23 * FDY3;
  }
  R DBTPDXA = R(0.5) * (DBTPDX1A + DBTPDX2A);   // Cfac1 = Cfac2 = 1
  R DBTPDYA = R(0.5) * (DBTPDY1A + DBTPDY2A);
  R ADVX = U1Avg * DU1DXA + V1Avg * DU1DYA;
  R ADVY = U1Avg * DV1DXA + V1Avg * DV1DYA;
  const Divisor<R, kFast> by_area(AreaIE, bad);
  R DU1DX = by_area(DU1DXA, bad), DU1DY = by_area(DU1DYA, bad);
  R DV1DX = by_area(DV1DXA, bad), DV1DY = by_area(DV1DYA, bad);
  const Divisor<R, kFast> by_h1(H1N1, bad), by_h2(H1N2, bad), by_h3(H1N3, bad);
  R EH1 = EVMEle * H1N1, EH2 = EVMEle * H1N2, EH3 = EVMEle * H1N3;
  R nc = (R)NCEle;
  R fct = nc * DT;
  R ax = -p.ifnlct * ADVX - GO2 * DBTPDXA - R(0.0);
  R ay = -p.ifnlct * ADVY - GO2 * DBTPDYA - R(0.0);
  R o[6];
  o[0] = fct * (ax - by_h1(R(1.5) * ((EH1 * DU1DX) * FDX1 + (EH1 * DU1DY) * FDY1), bad));
  o[1] = fct * (ax - by_h2(R(1.5) * ((EH2 * DU1DX) * FDX2 + (EH2 * DU1DY) * FDY2), bad));
  o[2] = fct * (ax - by_h3(R(1.5) * ((EH3 * DU1DX) * FDX3 + (EH3 * DU1DY) * FDY3), bad));
  o[3] = fct * (ay - by_h1(R(1.5) * ((EH1 * DV1DX) * FDX1 + (EH1 * DV1DY) * FDY1), bad));
  o[4] = fct * (ay - by_h2(R(1.5) * ((EH2 * DV1DX) * FDX2 + (EH2 * DV1DY) * FDY2), bad));
  o[5] = fct * (ay - by_h3(R(1.5) * ((EH3 * DV1DX) * FDX3 + (EH3 * DV1DY) * FDY3), bad));
  warp_store_k<6>(reinterpret_cast<R *>(c.ebuf) + 6 * (size_t)e0, o, nvalid, sh);
  return bad;
}

template <class R>
__device__ __forceinline__ void warp_mom(const adc_ctx &c, int e0, R *sh, bool alpha) {
  if constexpr (sizeof(R) == 8) {
    if (!__any_sync(0xffffffffu, warp_mom_by<R, true>(c, e0, sh, alpha))) return;
  }
  warp_mom_by<R, false>(c, e0, sh, alpha);
}

// gfortran's inline NORM2 for TKM(:,i) (scaled sum of squares starting
// from scale = 1), used by adcirc_norm2 (global.F:1502-1515).
__device__ inline double norm2_3(const double *x) {
  double scale = 1.0, result = 0.0;
  for (int i = 0; i < 3; ++i) {
    if (x[i] != 0.0) {
      double absx = fabs(x[i]);
      if (scale < absx) {
        double val = scale / absx;
        result = 1.0 + result * val * val;
        scale = absx;
      } else {
        double val = absx / scale;
        result = result + val * val;
      }
    }
  }
  return scale * sqrt(result);
}


// Nodal load, boundary condition and solve (momentum.F:713-1182).
template <class R, bool kFast>
__device__ __forceinline__ bool node_mom_by(const adc_ctx &c, int i) {
  bool bad = false;
  const adc_params_t &p = c.p;
  const double DTO2 = p.dt / 2.0;
  const R *eb = reinterpret_cast<const R *>(c.ebuf);
  R mxr = R(0.0), myr = R(0.0);
  const int q0 = c.n2e_ptr[i], q1 = c.n2e_ptr[i + 1];
  for (int qc = q0; qc < q1; qc += kGatherChunk) {
    int ek[kGatherChunk];
    R xa[kGatherChunk], xb[kGatherChunk];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k) if (qc + k < q1) ek[k] = c.n2e[qc + k];
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (qc + k < q1) {
        int e = ek[k] / 3, kk = ek[k] - 3 * e;
        xa[k] = eb[6 * (size_t)e + kk];
        xb[k] = eb[6 * (size_t)e + 3 + kk];
      }
#pragma unroll
    for (int k = 0; k < kGatherChunk; ++k)
      if (qc + k < q1) {
        mxr = mxr + xa[k];
        myr = myr + xb[k];
      }
  }
  double mx = (double)mxr, my = (double)myr;
  int NCI = c.nodecode[i];
  double ta = c.totalarea[i];
  if (ta != 0.0) {
    const Divisor<double, kFast> by(ta, bad);
    mx = by(mx, bad);
    my = by(my, bad);
  }
  double uu1 = c.uu1[i], vv1 = c.vv1[i];
  double WSX = 0.0, WSY = 0.0;
  if (p.nws != 0) {
    const Divisor<double, kFast> by_h1(c.h1[i], bad), by_h2(c.h2[i], bad);
    WSX = DTO2 * p.ifwind * (by_h1(c.wsx1[i], bad) + by_h2(c.wsx2[i], bad));
    WSY = DTO2 * p.ifwind * (by_h1(c.wsy1[i], bad) + by_h2(c.wsy2[i], bad));
  }
  const double *tkm = c.tkm + 3 * i;
  double VXX = DTO2 * (tkm[0] + 0.0);
  double VYY = DTO2 * (tkm[1] + 0.0);
  double CorifA = c.corif[i];
  double VXY = DTO2 * (tkm[2] - CorifA);
  double VYX = DTO2 * (tkm[2] + CorifA);
  mx = NCI * (mx + WSX + (1.0 - VXX) * uu1 - VXY * vv1);
  my = NCI * (my + WSY + (1.0 - VYY) * vv1 - VYX * uu1);
  double a1 = 1.0 + VXX * NCI, a2 = 1.0 + VYY * NCI, a3 = VXY * NCI, a4 = VYX * NCI;
  int me = c.me_of_node[i];
  if (me >= 0) {
    int lb = c.me_lbc[me];
    double csi = c.me_csi[me], sii = c.me_sii[me];
    const double qn2 = c.qn[2 * c.nvel + c.me_i[me]];   // zero on land boundaries
    if (lb >= 0 && lb <= 9) {
      double VelNorm = -qn2 / c.h2[i];
      if (fabs(norm2_3(tkm) - sqrt(2.0) * c.tk[i]) < DBL_EPSILON) {
        mx = (sii * mx - csi * my - VelNorm * a3) * NCI;
        my = VelNorm * a1 * NCI;
        a3 = -csi * a1;
        a4 = -a3;
        a1 = sii * a1;
        a2 = a1;
      } else {
        mx = (sii * mx - csi * my) * NCI;
        my = VelNorm * NCI;
        double n1 = a1 * sii - a4 * csi;
        double n3 = a3 * sii - a2 * csi;
        a1 = n1;
        a3 = n3;
        a4 = csi;
        a2 = sii;
      }
    }
    if (lb >= 10 && lb <= 19) {
      double VelNorm = -qn2 / c.h2[i];
      mx = 0.0 * NCI;
      my = VelNorm * NCI;
      a1 = sii;
      a3 = -csi;
      a4 = csi;
      a2 = sii;
    }
    if (lb == 41) {
      // zero normal velocity gradient by a Galerkin normal derivative over
      // the ring's elements (momentum.F:864-933), from the old velocities
      double r1 = 0.0, r2 = 0.0, lhs = 0.0;
      for (int q = c.me41_ptr[me]; q < c.me41_ptr[me + 1]; ++q) {
        const int nm2 = c.me41_tri[3 * q], nm3 = c.me41_tri[3 * q + 1], e = c.me41_tri[3 * q + 2];
        if (e < 0) continue;
        const int NCEle = NCI * c.nodecode[nm2] * c.nodecode[nm3] * c.noff[e];
        if (NCEle == 0) continue;
        const double FDX1 = c.fdx[3 * e] * 1.0, FDX2 = c.fdx[3 * e + 1] * 1.0, FDX3 = c.fdx[3 * e + 2] * 1.0;
        const double FDY1 = c.fdy[3 * e] * 1.0, FDY2 = c.fdy[3 * e + 1] * 1.0, FDY3 = c.fdy[3 * e + 2] * 1.0;
        r1 = r1 - (csi * FDX2 + sii * FDY2) * c.uu1[nm2] - (csi * FDX3 + sii * FDY3) * c.uu1[nm3];
        r2 = r2 - (csi * FDX2 + sii * FDY2) * c.vv1[nm2] - (csi * FDX3 + sii * FDY3) * c.vv1[nm3];
        lhs = lhs + csi * FDX1 + sii * FDY1;
      }
      if (NCI == 0) {
        mx = 0.0;
        my = 0.0;
      } else {
        mx = r1 / lhs;
        my = r2 / lhs;
      }
      a1 = 1.0;
      a2 = 1.0;
      a3 = 0.0;
      a4 = 0.0;
    }
  }
  c.mom_x[i] = mx;
  c.mom_y[i] = my;
  double DDU = a1 * a2 - a3 * a4;
  const Divisor<double, kFast> by_det(DDU, bad);
  double u2 = by_det(mx * a2 - my * a3, bad);
  double v2 = by_det(my * a1 - mx * a4, bad);
  c.uu2[i] = u2;
  c.vv2[i] = v2;
  double h2 = c.h2[i];
  c.qx2[i] = u2 * h2;
  c.qy2[i] = v2 * h2;
  return bad;
}

template <class R>
__device__ __forceinline__ void node_mom(const adc_ctx &c, int i) {
  if (node_mom_by<R, true>(c, i)) node_mom_by<R, false>(c, i);
}

// Zero normal velocity gradient (IBTYPE 40), momentum.F:1157-1174: after
// the nodal solve each such boundary node takes the velocity interpolated
// at its fictitious interior node, then its fluxes (:1179-1182).  The
// entries go in ME2GW order on one thread, since an entry's element may
// hold a node an earlier entry has just set.
__device__ inline void one_zng(const adc_ctx &c) {
  for (int k = 0; k < c.n_zng; ++k) {
    const int n = c.zng_node[k], e = c.zng_ele[k];
    const int NM1 = c.nm[3 * e], NM2 = c.nm[3 * e + 1], NM3 = c.nm[3 * e + 2];
    const int NCEle = c.nodecode[NM1] * c.nodecode[NM2] * c.nodecode[NM3] * c.noff[e];
    const double f1 = c.zng_f[3 * k], f2 = c.zng_f[3 * k + 1], f3 = c.zng_f[3 * k + 2];
    const double u = NCEle * (c.uu2[NM1] * f1 + c.uu2[NM2] * f2 + c.uu2[NM3] * f3);
    const double v = NCEle * (c.vv2[NM1] * f1 + c.vv2[NM2] * f2 + c.vv2[NM3] * f3);
    c.uu2[n] = u;
    c.vv2[n] = v;
    c.qx2[n] = u * c.h2[n];
    c.qy2[n] = v * c.h2[n];
  }
}

// End of a step of adc_run: the iteration log and the step table's cursor.
__device__ __forceinline__ void step_end(const adc_ctx &c, int *log, int cap) {
  const int k = c.flags->cursor;
  if (k < cap) log[k] = c.flags->numitr;
  c.flags->cursor = k + 1;
}

}  // namespace adc
