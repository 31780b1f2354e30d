// jcg_ordered.cu -- ITPACK 2D JCG for the modes with FP32 parts, and in FP64
// for matrices beyond the resident kernel (jcg_resident.cu).
//
// In the modes with FP32 parts a last-bit change of a dot product changes, now and then,
// how a value rounds to FP32, and from there a run's results at the 1e-6
// level.  This kernel therefore keeps the summation tree those modes have
// always had (256-thread row blocks, their block sums in block order), where
// jcg_resident.cu, with its larger blocks, has another.
//
//  * Two row blocks per SM of about 2,048 rows, plus one scalar block.  A
//    row block keeps dtwd, d(in) and d(in-1) of its rows in shared memory
//    and streams the scaled matrix (FP32 with ADC_F32_SPMV, FP64 products)
//    through per-warp double buffers of bulk copies.
//  * One grid barrier per iteration: a halo row's new d is formed from its
//    owner's exported (dtwd, d, d(in-1)) record by the owner's expression.
//  * The scalar block's first warp computes chgcon while the rows work.
//  * Every wait is bounded (clock64); on expiry the kernel records a timeout
//    and all blocks return.
#include "jcg_grid.cuh"
#include "jcg_scalar.cuh"
#include "tma.cuh"

#include <cfloat>
#include <cstring>
#include <type_traits>
#include <vector>
#include <algorithm>

namespace adc {

constexpr int kRowUnroll = 8;   // rows per thread whose loads issue together
constexpr int kHaloPre = 2;     // halo records per thread fetched ahead of the row update

// Per-warp double-buffered bulk copies of whole slices (block-local
// columns + one value array) into shared memory.
// Every copy that is issued is waited for before the next phase.
struct SlicePipe {
  unsigned char *stg0;        // this warp's two buffers
  uint64_t *bar0;             // and their mbarriers
  const int2 *meta;           // per slice of the block: (first slot, width)
  const unsigned short *lcol;
  Flags *flags;
  int stage_bytes, s0, s1, first, step, lane;
  uint32_t parbits;
  int wcap;                   // slices wider than this are not staged
  long long spin;             // cycles a wait may take

  __device__ bool staged(int sl) const { return meta[sl - s0].y <= wcap; }

  // V: the staged value type (FP64 matrix, or FP32 in the mixed mode)
  template <class V>
  __device__ void issue(int sl, int st, const V *vals) {
    if (lane == 0 && staged(sl)) {
      const int2 mt = meta[sl - s0];
      const uint32_t w = (uint32_t)mt.y;
      const uint32_t vb = w * 32u * (uint32_t)sizeof(V);
      unsigned char *b = stg0 + (size_t)st * stage_bytes;
      mbar_expect_tx(bar0 + st, w * 64u + vb);
      if (w > 0) {
        bulk_load(b, lcol + mt.x, w * 64u, bar0 + st);
        bulk_load(b + w * 64u, vals + mt.x, vb, bar0 + st);
      }
    }
  }
  // Starts the warp's first two slices; with `fence`, first orders earlier
  // generic writes of `vals` before the copies.
  template <class V>
  __device__ void begin(const V *vals, bool fence) {
    if (fence && lane == 0) fence_proxy_async_all();
    if (first < s1) issue(first, 0, vals);
    if (first + step < s1) issue(first + step, 1, vals);
  }
  // Waits for a copy in flight for kDrainCycles more.
  __device__ void drain(int st) {
    const long long tw = clock64();
    while (!mbar_try_wait(bar0 + st, (parbits >> st) & 1u) && clock64() - tw < kDrainCycles) {
    }
  }
  // The answer is the warp's: lanes that look at the clock one by one may
  // differ.
  __device__ bool wait(int st, bool other_in_flight) {
    const long long tw = clock64();
    bool ok;
    while (!(ok = mbar_try_wait(bar0 + st, (parbits >> st) & 1u)) && clock64() - tw <= spin) {
    }
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) {
        atomicExch(&flags->timeout, 1);
        // let this copy and the one already issued into the other buffer land
        drain(st);
        if (other_in_flight) drain(st ^ 1);
      }
      __syncwarp();
      return false;
    }
    parbits ^= 1u << st;
    return true;
  }
  // body(sl, lc, lv): one slice from shared memory (or, for a slice wider
  // than wcap, in place from global memory, which has the same layout);
  // lc/lv hold slot q of lane l at [q * 32 + l].  Returns false on an
  // expired wait.
  template <class V, class F>
  __device__ bool run(const V *vals, F body) {
    int k = 0;
    for (int sl = first; sl < s1; sl += step, ++k) {
      const int st = k & 1;
      const int2 mt = meta[sl - s0];
      if (mt.y > wcap) {
        body(sl, lcol + mt.x, vals + mt.x);
      } else {
        if (!wait(st, sl + step < s1 && staged(sl + step))) return false;
        const unsigned char *b = stg0 + (size_t)st * stage_bytes;
        body(sl, (const unsigned short *)b, (const V *)(b + (size_t)mt.y * 64));
      }
      __syncwarp();
      if (sl + 2 * step < s1) issue(sl + 2 * step, st, vals);
    }
    return true;
  }
};

// VT: storage type of the scaled matrix the iterations stream.
template <class VT>
__global__ void __launch_bounds__(kThreads, 2) jcg_ordered_kernel(JcgArgs a) {
  griddep_wait();
  VT *const sv_store = std::is_same<VT, float>::value ? (VT *)a.soff32 : (VT *)a.soff;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const bool scalar_block = (blockIdx.x == (unsigned)a.nrb);
  const int s0 = scalar_block ? 0 : (int)((long long)a.nslices * blockIdx.x / a.nrb);
  const int s1 = scalar_block ? 0 : (int)((long long)a.nslices * (blockIdx.x + 1) / a.nrb);
  const int n = a.n;
  const int r0 = s0 * kSlice, rows = (s1 - s0) * kSlice;   // the block's rows [r0, r0 + rows)
  extern __shared__ __align__(128) unsigned char s_dyn[];
  // Dynamic shared memory.  Scalar block: the CG tridiagonal.  Row blocks:
  // dtwd of the block's rows; two value buffers
  // (d of the rows, then the halo's new d) that trade roles every
  // iteration; per row its length and export bit; the slice table; one
  // mbarrier and two staging buffers per warp.
  double2 *const tri = (double2 *)s_dyn;
  P4 *const p0 = (P4 *)a.p0, *const p1 = (P4 *)a.p1;
  const int RB = a.rows_max, VB = a.rows_max + a.halo_max;
  double *S_t = (double *)s_dyn;
  double *S_dd = S_t + RB;
  unsigned char *S_le = (unsigned char *)(S_dd + 2 * VB);
  int2 *S_meta = (int2 *)(S_le + ((RB + 127) & ~127));
  int *S_hid = (int *)(S_meta + ((RB / kSlice + 15) & ~15));   // the block's halo nodes
  uint64_t *S_bar = (uint64_t *)(S_hid + ((a.halo_max + 31) & ~31));
  unsigned char *S_stage = (unsigned char *)(S_bar + 16);
  const int nhalo = !scalar_block ? a.halo_ptr[blockIdx.x + 1] - a.halo_ptr[blockIdx.x] : 0;
  SlicePipe pipe{S_stage + (size_t)(2 * warp) * a.stage_bytes, &S_bar[2 * warp], S_meta, a.lcol,
                 a.flags, a.stage_bytes, s0, s1, s0 + warp, nwarps, lane, 0u, a.stage_wcap, a.spin};
  __shared__ ItpLocal L;              // used by the scalar block's thread 0 only
  __shared__ Rec s_rec;               // the record of the last reducing barrier
  unsigned gen = a.bar->gen;          // barrier generation, going on from solve to solve
  const int q1 = a.itp->q1;
  if (threadIdx.x == 0) {
    // Every block steps its own copy of the ITPACK scalars, from echall's
    // start of a solve (itpackv.F:1212-1255, the zeta floor of jcg :223-232)
    // or, without run_init, from the caller's: cme is the last solve's until
    // chgcon(0), q1 and rparm1 stay.
    const volatile Itp *g = a.itp;
    L.rparm1 = g->rparm1;
    L.zeta = a.run_init ? L.rparm1 : g->zeta;
    if (a.run_init && L.zeta < 512.0 * DBL_EPSILON) L.zeta = 512.0 * DBL_EPSILON;
    L.cme = g->cme;
    L.cmold = g->cmold;
    L.gamold = g->gamold;
    L.rhoold = g->rhoold;
    L.delnnm = L.delsnm = L.gamma = L.rho = L.stptst = L.udnm = 0.0;
    L.itmax = a.itmax; L.adapt = a.run_init ? 1 : g->adapt; L.q1 = q1; L.isym = 0; L.chg_ier = 0;
  }
  __syncthreads();

  const double ztol = scalar_block && warp == 0 ? zbrent_tol(L.zeta) : 0.0;
  // chgcon for iteration `in` in the scalar block's first warp, from the
  // scalars the last exchange left in L.
  auto estimate = [&](int in) {
    if (warp != 0) return;
    double cme = L.cme, cmold = L.cmold;
    int adapt = L.adapt, ier = L.chg_ier;
    if (adapt) chgcon_warp<true>(L.gamma, L.rho, L.gamold, L.rhoold, L.zeta, ztol, a.itmax, tri, in, cme, cmold, adapt, ier);
    __syncwarp();
    if (lane == 0) {
      L.cme = cme;
      L.cmold = cmold;
      L.adapt = adapt;
      L.chg_ier = ier;
    }
    __syncwarp();
  };

  const int need_u0 = !q1;   // the norm of u at iteration 0
  double pd = 0.0, pt = 0.0, pu = 0.0;
  // Prologue.  Shared memory first holds, per row of the block
  // and per halo node, w = 1/sqrt(diag) and u' (P1), then d0 (P2).
  double *Uv = S_dd, *Wv = S_dd + VB;
  if (!scalar_block) {
    // Everything the prologue needs from global memory is requested
    // before any of it is stored, so the loads share one round trip: the
    // slice table, the halo list, and per row its length, export bit and
    // the diagonal, u and rhs of P0 (scal part 1: u' = u*sqrt(d),
    // w = 1/sqrt(d), rhs' = rhs*w).
    const int nsl = s1 - s0;
    const int h0 = a.halo_ptr[blockIdx.x];
    int2 mt = make_int2(0, 0);
    if ((int)threadIdx.x < nsl) mt = make_int2(a.sl_ptr[s0 + threadIdx.x], a.sl_w[s0 + threadIdx.x]);
    int hid[kHaloPre];
#pragma unroll
    for (int k = 0; k < kHaloPre; ++k) {
      const int h = threadIdx.x + k * blockDim.x;
      hid[k] = h < nhalo ? a.halo_ids[h0 + h] : 0;
    }
    for (int base = threadIdx.x; base < rows; base += kRowUnroll * blockDim.x) {
      double dg[kRowUnroll], uu[kRowUnroll], rh[kRowUnroll];
      int rl[kRowUnroll];
      unsigned char ex[kRowUnroll];
#pragma unroll
      for (int k = 0; k < kRowUnroll; ++k) {
        const int idx = base + k * blockDim.x, i = r0 + idx;
        if (idx < rows && i < n) {
          dg[k] = a.diag[i]; uu[k] = a.u[i]; rh[k] = a.rhs[i];
          rl[k] = a.rlen[i]; ex[k] = a.exp[i];
        }
      }
#pragma unroll
      for (int k = 0; k < kRowUnroll; ++k) {
        const int idx = base + k * blockDim.x, i = r0 + idx;
        if (idx < rows) S_le[idx] = i < n ? (unsigned char)(rl[k] | (ex[k] ? 128 : 0)) : 0;
        if (idx < rows && i < n) {
          double work = sqrt(dg[k]);
          const double up = uu[k] * work;
          double wv = 1.0 / work;
          a.u1[i] = up;   // u' goes to u1: u keeps the raw guess until P2
          a.w[i] = wv;
          a.rhs[i] = rh[k] * wv;
          Uv[idx] = up;
          Wv[idx] = wv;
          if (need_u0) pu += up * up;
        }
      }
    }
    if ((int)threadIdx.x < nsl) S_meta[threadIdx.x] = mt;
    for (int k = threadIdx.x + blockDim.x; k < nsl; k += blockDim.x)
      S_meta[k] = make_int2(a.sl_ptr[s0 + k], a.sl_w[s0 + k]);
#pragma unroll
    for (int k = 0; k < kHaloPre; ++k) {
      const int h = threadIdx.x + k * blockDim.x;
      if (h < nhalo) S_hid[h] = hid[k];
    }
    for (int h = threadIdx.x + kHaloPre * blockDim.x; h < nhalo; h += blockDim.x)
      S_hid[h] = a.halo_ids[h0 + h];
    if (threadIdx.x < 2 * nwarps) mbar_init(&S_bar[threadIdx.x], 1);
    mbar_fence_init();
  }
  // No grid barrier after P0: P1 reads only this block's own P0 results,
  // and forms the halo's u' and w itself from the raw u and diag, which
  // no block overwrites before P2.
  __syncthreads();
  // P1: scaled off-diagonals, the reference's unscal drift of the resident
  // matrix, and d0 = pjac(u') + rhs' - u' (kept in S_t until P2).
  if (!scalar_block) {
    pipe.begin(a.offd, false);   // offd was last written by an earlier kernel
    const int nh = nhalo;
    for (int h = threadIdx.x; h < nh; h += blockDim.x) {
      const int j = S_hid[h];
      double work = sqrt(a.diag[j]);   // the owner's P0 expressions
      Uv[RB + h] = a.u[j] * work;
      Wv[RB + h] = 1.0 / work;
    }
    __syncthreads();
    bool ok = pipe.run(a.offd, [&](int sl, const unsigned short *lc, const double *lv) {
      const int i = sl * kSlice + lane, idx = i - r0;
      if (i < n) {
        const int len = S_le[idx] & 127;
        const int base = S_meta[sl - s0].x + lane;
        const double wi = Wv[idx], ui = Uv[idx];
        const double winv_i = 1.0 / wi;
        double acc = a.rhs[i];
        for (int q = 0; q < len; ++q) {
          const int lq = lc[q * kSlice + lane];
          const double wj = Wv[lq];
          const double sv = lv[q * kSlice + lane] * wi * wj;
          sv_store[base + q * kSlice] = (VT)sv;
          if (!a.defer_drift) a.offd[base + q * kSlice] = sv * winv_i * (1.0 / wj);
          acc = acc - sv * Uv[lq];
        }
        const double d0 = acc - ui;
        if (S_le[idx] & 128) st_p4(p0 + i, 0.0, d0, 0.0, 0.0);
        S_t[idx] = d0;
      }
    });
    if (!ok) atomicExch(&a.flags->timeout, 1);
    fence_proxy_async_all();   // soff is read by bulk copies from here on
  }
  if (!phase_sync(a, scalar_block, gen)) return;
  // P2: dtwd0 = -A' d0 and the iteration-0 norms.
  if (!scalar_block) {
    pipe.begin((const VT *)sv_store, true);   // the scaled matrix was just written
    double *Dv = S_dd;
    for (int idx = threadIdx.x; idx < rows; idx += blockDim.x) {
      Dv[idx] = S_t[idx];
      S_dd[VB + idx] = 0.0;   // d(-1)
      const int i = r0 + idx;
      if (i < n) {
        // every block has read the raw u and diag by now (the P1 barrier)
        a.u[i] = 0.0;   // u(-1) of the recurrence
        const double winv_i = 1.0 / a.w[i];
        a.diag[i] = winv_i * winv_i;   // scal/unscal of the diagonal
      }
    }
    const int nh = nhalo;
    for (int h = threadIdx.x; h < nh; h += blockDim.x) Dv[RB + h] = p0[S_hid[h]].y;
    __syncthreads();
    bool ok = pipe.run((const VT *)sv_store, [&](int sl, const unsigned short *lc, const VT *lv) {
      const int i = sl * kSlice + lane, idx = i - r0;
      if (i < n) {
        const int len = S_le[idx] & 127;
        double acc = 0.0;
        for (int q = 0; q < len; ++q)
          acc = acc - (double)lv[q * kSlice + lane] * Dv[lc[q * kSlice + lane]];
        if (S_le[idx] & 128) p0[i].x = acc;
        S_t[idx] = acc;
        const double di = Dv[idx];
        pd += di * di;
        pt += di * acc;
      }
    });
    if (!ok) atomicExch(&a.flags->timeout, 1);
  }
  {
    if (scalar_block) estimate(0);
    const int need_u = need_u0;
    bool ok = phase_reduce(a, scalar_block, gen, pd, pt, pu, L.cme,
                           [&](double sd, double st, double su, double cme) {
      L.cme = cme;   // chgcon's estimate, from the scalar block
      L.delnnm = sd;
      int halt = pstop_d(&L, 0, need_u ? su : 1.0, sd);
      double c[4] = {0, 0, 0, 0};
      if (!halt) {
        if (L.itmax == 0) halt = 2;
        else parcon_d(&L, 0, st, c);
      }
      Rec *vr = &s_rec;
      vr->c1 = c[0]; vr->c2 = c[1]; vr->c3 = c[2]; vr->c4 = c[3];
      vr->halt = halt;
      vr->need_unorm = !(L.q1 || ((1 > 5) && (1 % 5 != 0)));
      vr->in = 0;
    });
    if (!ok) return;
  }

  // Iteration phases: phase `in` forms u(in+1), d(in+1), dtwd(in+1) and the
  // norms of iteration in+1.  P[in % 2][i] = (dtwd(in), d(in), d(in-1)) so
  // a neighbour's three values arrive in one 32-byte sector.
  P4 *P[2] = {p0, p1};
  // u(in) and u(in-1): the prologue leaves u' in u1 and zeroes u
  double *U[2] = {a.u1, a.u};
  int cur = 0;   // S_dd half holding d(in)
  for (int in = 0; in < a.itmax; ++in) {
    const Rec r = s_rec;
    if (r.halt) break;
    const double c1 = r.c1, c2 = r.c2, c3 = r.c3, c4 = r.c4;
    const int need_u = r.need_unorm;
    const P4 *pc = P[in % 2];
    P4 *pn = P[(in + 1) % 2];
    const double *uc = U[in % 2];
    double *un = U[(in + 1) % 2];
    double pd = 0.0, pt = 0.0, pu = 0.0;
    if (!scalar_block) {
      // The warp's first two slices start streaming before phase A.
      pipe.begin((const VT *)sv_store, false);   // unchanged since P2's fence
      // Phase A: the 3-term update of the block's rows, d(in+1) written
      // over d(in-1); then the new d of the halo nodes from their owners'
      // exported records (same expression, same bits).
      double *Sd = S_dd + cur * VB, *Sdn = S_dd + (cur ^ 1) * VB;
      const int nh = nhalo;
      P4 hv[kHaloPre];   // the first halo records, loaded with the rows' vectors
#pragma unroll
      for (int k = 0; k < kHaloPre; ++k) {
        const int h = threadIdx.x + k * blockDim.x;
        if (h < nh) hv[k] = ld_p4(pc + S_hid[h]);
      }
      for (int base = threadIdx.x; base < rows; base += kRowUnroll * blockDim.x) {
        double ucv[kRowUnroll], unv[kRowUnroll];
#pragma unroll
        for (int k = 0; k < kRowUnroll; ++k) {
          const int idx = base + k * blockDim.x, i = r0 + idx;
          if (idx < rows && i < n) { ucv[k] = uc[i]; unv[k] = un[i]; }
        }
#pragma unroll
        for (int k = 0; k < kRowUnroll; ++k) {
          const int idx = base + k * blockDim.x, i = r0 + idx;
          if (idx < rows && i < n) {
            const double dn = c1 * S_t[idx] + c4 * Sd[idx] + c3 * Sdn[idx];
            const double unew = c1 * Sd[idx] + c2 * ucv[k] + c3 * unv[k];
            Sdn[idx] = dn;
            un[i] = unew;
            if (need_u) pu += unew * unew;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kHaloPre; ++k) {
        const int h = threadIdx.x + k * blockDim.x;
        if (h < nh) Sdn[RB + h] = c1 * hv[k].x + c4 * hv[k].y + c3 * hv[k].z;
      }
      for (int h = threadIdx.x + kHaloPre * blockDim.x; h < nh; h += blockDim.x) {
        const P4 o = ld_p4(pc + S_hid[h]);
        Sdn[RB + h] = c1 * o.x + c4 * o.y + c3 * o.z;
      }
      __syncthreads();
      // Phase B: the SpMV from shared memory, slot order as in pjac.
      bool ok = pipe.run((const VT *)sv_store, [&](int sl, const unsigned short *lc, const VT *lv) {
        const int i = sl * kSlice + lane, idx = i - r0;
        if (i < n) {
          const unsigned le = S_le[idx];
          const int len = (int)(le & 127u);
          double acc = 0.0;
#pragma unroll 4
          for (int q = 0; q < len; ++q)
            acc = acc - (double)lv[q * kSlice + lane] * Sdn[lc[q * kSlice + lane]];
          const double dn = Sdn[idx];
          if (le & 128u) st_p4(pn + i, acc, dn, Sd[idx], 0.0);
          S_t[idx] = acc;
          pd += dn * dn;
          pt += dn * acc;
        }
      });
      if (!ok) atomicExch(&a.flags->timeout, 1);
      cur ^= 1;
    }
    const int m = in + 1;
    if (scalar_block) estimate(m);
    bool ok = phase_reduce(a, scalar_block, gen, pd, pt, pu, L.cme,
                           [&](double sd, double st, double su, double cme) {
      L.cme = cme;   // chgcon's estimate, from the scalar block
      L.delnnm = sd;
      int halt = pstop_d(&L, m, need_u ? su : 1.0, sd);
      double c[4] = {0, 0, 0, 0};
      if (!halt) {
        if (m >= L.itmax) halt = 2;
        else parcon_d(&L, m, st, c);
      }
      int mm = m + 1;
      Rec *vr = &s_rec;
      vr->c1 = c[0]; vr->c2 = c[1]; vr->c3 = c[2]; vr->c4 = c[3];
      vr->halt = halt;
      vr->need_unorm = !(L.q1 || ((mm > 5) && (mm % 5 != 0)));
      vr->in = m;
    });
    if (!ok) return;
  }
  const Rec r = s_rec;
  const int fin = r.in;
  const double *usol = U[fin % 2];

  // Epilogue: unscal (itpackv.F:2447-2477), the GWCE eta update
  // (gwce.F:2006-2008) and wet/dry pass D1.
  for (int s = s0 + warp; s < s1; s += nwarps) {
    int i = s * kSlice + lane;
    if (i < n) {
      double wv = a.w[i];
      const double us = usol[i];
      double uf = us * wv;
      if (a.do_peror) {   // scaled u and rhs for jcg_peror_kernel; the records are done with
        a.u1[i] = us;
        ((double *)a.p0)[2 * (size_t)a.nslices * kSlice + i] = a.rhs[i];
      }
      a.u[i] = uf;
      a.rhs[i] = a.rhs[i] * (1.0 / wv);
      if (a.eta_update) {
        const int nc = a.nodecode[i];
        double e2 = nc * (uf + 0.0) + a.eta1[i];
        if (a.d1 && d1_dries(nc, a.dp[i], a.h0, e2)) {
          a.nnodecode[i] = 0;
          a.nodecode[i] = 0;
          atomicAdd(&a.flags->ncchange, 1);
        }
        a.eta2[i] = e2;
      }
    }
  }
  if (scalar_block && threadIdx.x == 0) {
    int h = r.halt;
    if (h == 2) L.rparm1 = L.stptst;   // itpackv.F:394
    volatile Itp *g = a.itp;
    g->zeta = L.zeta; g->cme = L.cme; g->gamma = L.gamma; g->rho = L.rho;
    g->gamold = L.gamold; g->rhoold = L.rhoold; g->delnnm = L.delnnm; g->delsnm = L.delsnm;
    g->udnm = L.udnm; g->stptst = L.stptst; g->cmold = L.cmold; g->rparm1 = L.rparm1;
    g->sme = -1.0; g->itmax = L.itmax; g->isym = 0;
    g->adapt = L.adapt; g->q1 = L.q1; g->chg_ier = L.chg_ier;
    g->in = fin;
    g->halt = h;
    a.bar->gen = gen;
    if (a.est) a.est->exact = 1;
    if (a.d1) a.flags->n_w1_events = 0;
    if (a.defer_drift == 1) *a.drift_pending = 1;
    a.flags->numitr = fin;
    a.flags->ier = (h == 2) ? 13 : 0;
    a.flags->zeta = L.rparm1;
    a.flags->cme = L.cme;
  }
}

static size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }

static size_t jcg_stage_bytes(int wmax) { return round_up((size_t)std::max(wmax, 1) * 320, 128); }

// Dynamic shared memory of one block (the largest of the scalar block's
// tridiagonal and a row block's layout, see the kernel).
static size_t jcg_smem_bytes(int itmax, int rows_max, int halo_max, int wmax) {
  size_t tri = round_up(sizeof(double2) * (itmax + 2), 128);
  size_t rb = (size_t)rows_max, vb = rb + (size_t)halo_max;
  size_t rowb = 8 * rb + 16 * vb + round_up(rb, 128) + 8 * round_up(rb / kSlice, 16) +
                4 * round_up((size_t)halo_max, 32) + 128 + 16 * jcg_stage_bytes(wmax);
  return std::max(tri, rowb);
}

static int jcg_row_block_begin(int nslices, int nrb, int b) {
  return (int)((long long)nslices * b / nrb);
}

// Block-local column indices.  Row block b owns the
// rows of slices [s0, s1); a neighbour in that range maps to its offset
// from the block's first row, any other neighbour to rows_max + its
// position in the block's halo list (first appearance in slot order).
// exp[j] = 1 marks rows that another block reads.
static void jcg_local_tables(int n, int nslices, int nrb, int rows_max, const int *sl_ptr,
                             const int *sl_w, const int *col, const int *rlen,
                             std::vector<unsigned short> &lcol, std::vector<int> &halo_ptr,
                             std::vector<int> &halo_ids, std::vector<unsigned char> &exp,
                             int &halo_max) {
  lcol.assign(std::max(sl_ptr[nslices], 1), 0);
  halo_ptr.assign(nrb + 1, 0);
  halo_ids.clear();
  exp.assign((size_t)nslices * kSlice, 0);
  std::vector<int> stamp(n, -1), hid(n, 0);
  halo_max = 0;
  for (int b = 0; b < nrb; ++b) {
    const int s0 = jcg_row_block_begin(nslices, nrb, b), s1 = jcg_row_block_begin(nslices, nrb, b + 1);
    const int r0 = s0 * kSlice, rows = (s1 - s0) * kSlice;
    int nh = 0;
    for (int sl = s0; sl < s1; ++sl)
      for (int k = 0; k < sl_w[sl]; ++k)
        for (int lane = 0; lane < kSlice; ++lane) {
          const int i = sl * kSlice + lane;
          if (i >= n || k >= rlen[i]) continue;
          const size_t q = (size_t)sl_ptr[sl] + (size_t)k * kSlice + lane;
          const int j = col[q];
          if (j >= r0 && j < r0 + rows) {
            lcol[q] = (unsigned short)(j - r0);
            continue;
          }
          if (stamp[j] != b) {
            stamp[j] = b;
            hid[j] = nh++;
            halo_ids.push_back(j);
            exp[j] = 1;
          }
          lcol[q] = (unsigned short)(rows_max + hid[j]);
        }
    halo_ptr[b + 1] = halo_ptr[b] + nh;
    halo_max = std::max(halo_max, nh);
  }
}

// Chooses the launch shape, builds the block-local tables and uploads them;
// done = false where this kernel does not apply.
int plan_jcg_ordered(adc_ctx *c, const JcgHostSell *h, int nsm, bool &done) {
  done = false;
  // keep at least ~8 slices per block so the barrier cost stays amortised
  int nrb0 = std::max(1, std::min(2 * nsm - 1, std::max(1, c->nslices / 8)));
  if (c->jcg_nrb_req > 0) nrb0 = std::max(1, std::min({c->jcg_nrb_req, 2 * nsm - 1, c->nslices}));
  const int nrb = nrb0;
  const int rows_max = (c->nslices + nrb - 1) / nrb * kSlice;
  int wmax = 1;
  for (int sl = 0; sl < c->nslices; ++sl) wmax = std::max(wmax, h->sl_w[sl]);
  std::vector<unsigned short> lcol;
  std::vector<int> hptr, hids;
  std::vector<unsigned char> exp;
  int halo_max = 0;
  bool fits = wmax < 128;
  if (fits) {
    jcg_local_tables(c->np, c->nslices, nrb, rows_max, h->sl_ptr, h->sl_w, h->col, h->rlen,
                     lcol, hptr, hids, exp, halo_max);
    fits = rows_max + halo_max < 65536;
  }
  // Stage slices up to width wcap in shared memory; a few wider slices
  // (rows with the most neighbours) are read in place, so that two row
  // blocks still fit on an SM.
  size_t smem = 0;
  int per_sm = 0, wcap = wmax;
  const void *fn = f32_spmv(c) ? (const void *)jcg_ordered_kernel<float>
                               : (const void *)jcg_ordered_kernel<double>;
  for (; fits && wcap >= std::max(1, wmax - 4); --wcap) {
    smem = jcg_smem_bytes(c->itmax, rows_max, halo_max, wcap);
    if (smem > 200 * 1024) continue;
    if (int rc = jcg_smem_limit(fn)) return rc;
    ADC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, smem));
    if (per_sm >= 2) break;
  }
  if (per_sm >= 2 && (long long)per_sm * nsm >= nrb + 1) {
    JcgTables T;
    const size_t o_lcol = T.add(lcol), o_hptr = T.add(hptr), o_hids = T.add(hids), o_exp = T.add(exp);
    if (int rc = T.upload(c)) return rc;
    c->jlcol = (unsigned short *)(c->jtab + o_lcol);
    c->jhalo_ptr = (int *)(c->jtab + o_hptr);
    c->jhalo_ids = (int *)(c->jtab + o_hids);
    c->jrle = c->jtab + o_exp;
    c->jcg_rows_blocks = nrb;
    c->jcg_grid = nrb + 1;
    c->jcg_res = 3;
    c->jcg_rows_max = rows_max;
    c->jcg_halo_max = halo_max;
    c->jcg_stage_bytes = (int)jcg_stage_bytes(wcap);
    c->jcg_stage_wcap = wcap;
    c->jcg_smem = smem;
    done = true;
    return ADC_OK;
  }
  return ADC_OK;
}

int launch_jcg_ordered(const JcgArgs &a0, const adc_ctx *c) {
  JcgArgs a = a0;
  a.rows_max = c->jcg_rows_max;
  a.halo_max = c->jcg_halo_max;
  a.stage_bytes = c->jcg_stage_bytes;
  a.stage_wcap = c->jcg_stage_wcap;
  a.lcol = c->jlcol;
  a.halo_ptr = c->jhalo_ptr;
  a.halo_ids = c->jhalo_ids;
  a.exp = c->jrle;
  const void *fn = f32_spmv(c) && c->soff32 ? (const void *)jcg_ordered_kernel<float>
                                             : (const void *)jcg_ordered_kernel<double>;
  void *args[] = {&a};
  ADC_CUDA(cudaLaunchCooperativeKernel(fn, dim3(c->jcg_grid), dim3(kThreads), args, c->jcg_smem, c->stream));
  return ADC_OK;
}

}  // namespace adc
