// jcg.cu -- ITPACK 2D JCG (itpackv.F:63-604) as one persistent cooperative
// kernel with its vectors in global memory, and the solver's set-up and
// launch.  Two kernels with block-local tables come first: jcg_resident.cu,
// where a matrix fits on the SMs (639,360 rows at most), then jcg_ordered.cu
// (about a million).  This one serves what neither takes (more rows, 128 or
// more neighbours, many wide rows together with a large ITMAX) and
// adc_jcg_noalloc, which builds no host tables.
//
// Design
//  * The scaled system (scal, itpackv.F:2281-2421) is built in-kernel from
//    the resident GWCE matrix, which also receives the reference's
//    scal/unscal rounding drift (itpackv.F:2447-2477) so a following solve
//    without a rebuild starts from the same bits.
//  * Each CG iteration is ONE grid-wide phase: a block updates u/d for its
//    rows (the 3-term recurrence, itpackv.F:593-596) and immediately forms
//    the next pseudo-residual SpMV (pjac, itpackv.F:1932-1967).  Neighbour
//    values of the new d are recomputed from the three previous buffers
//    (d rotates over 3 buffers, dtwd over 2) instead of waiting for their
//    owners, so the only grid barrier per iteration is the one the dot
//    products need.  The recomputation evaluates the same expression as
//    the owner, so every row sees identical bits.
//  * The dot products (sdot, itpackv.F:2828) are FP64 warp/block trees with
//    a fixed shape; every block sums the block partials in one fixed order
//    and runs the scalar ITPACK steps (pstop_nrms :809-890, parcon
//    :1774-1851) itself.
//  * The adaptive eigenvalue estimate (chgcon :893-1027 with zbrent/determ)
//    only feeds the stopping test and depends only on the previous
//    iteration's scalars, so a dedicated extra block computes it while the
//    others run the SpMV, taking its latency off the critical path.
//  * Every barrier wait is bounded (clock64); on expiry the kernel records
//    a timeout and all blocks return.
#include "jcg_grid.cuh"

#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>
#include <algorithm>

namespace adc {

// ------------------------------------------------------------ row access
// A row's off-diagonal slots are processed in chunks of kCh: the column and
// value of every slot of the chunk are loaded first, then all neighbour
// values are gathered, so the loads of a chunk are in flight together.
// Accumulation keeps the slot order (pjac's j order).
constexpr int kCh = 6;

// L2 prefetch of the next slice of a warp: the column and value rows of its
// slots and its own-row vector entries, one 128-byte line per lane.
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ void prefetch_slice(int lane, int ptr, int w, int row0, const int *col,
                                               const double *val, const P4 *pv,
                                               const double *u0, const double *u1) {
  // lines: col w, val 2w, pv 8, u0 2, u1 2
  const int ncol = w, nval = 2 * w;
  for (int l = lane; l < ncol + nval + 12; l += 32) {
    const char *a;
    if (l < ncol) a = (const char *)(col + ptr) + 128 * l;
    else if (l < ncol + nval) a = (const char *)(val + ptr) + 128 * (l - ncol);
    else if (l < ncol + nval + 8) a = (const char *)(pv + row0) + 128 * (l - ncol - nval);
    else if (l < ncol + nval + 10) a = (const char *)(u0 + row0) + 128 * (l - ncol - nval - 8);
    else a = (const char *)(u1 + row0) + 128 * (l - ncol - nval - 10);
    prefetch_l2(a);
  }
}

// ------------------------------------------------------------ the kernel
__global__ void __launch_bounds__(kThreads, 2) jcg_kernel(JcgArgs a) {
  griddep_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const bool scalar_block = (blockIdx.x == (unsigned)a.nrb);
  const int s0 = scalar_block ? 0 : (int)((long long)a.nslices * blockIdx.x / a.nrb);
  const int s1 = scalar_block ? 0 : (int)((long long)a.nslices * (blockIdx.x + 1) / a.nrb);
  const int n = a.n;
  extern __shared__ __align__(128) unsigned char s_dyn[];
  // Dynamic shared memory: tri(:,1) and tri(:,2) of the scalar block.
  double *t1 = (double *)s_dyn, *t2 = t1 + a.itmax + 1;
  P4 *const p0 = (P4 *)a.p0, *const p1 = (P4 *)a.p1;
  Rec *rec = &a.itp->rec;
  __shared__ ItpLocal L;              // used by the scalar block's thread 0 only
  __shared__ Rec s_rec;               // the record of the last reducing barrier
  unsigned gen = 0;                   // barrier generation within this launch
  if (threadIdx.x == 0) {   // every block steps its own copy of the ITPACK scalars
    const volatile Itp *g = a.itp;
    L.zeta = g->zeta; L.cme = g->cme; L.gamma = g->gamma; L.rho = g->rho;
    L.gamold = g->gamold; L.rhoold = g->rhoold; L.delnnm = g->delnnm; L.delsnm = g->delsnm;
    L.udnm = g->udnm; L.stptst = g->stptst; L.cmold = g->cmold; L.rparm1 = g->rparm1;
    L.itmax = g->itmax; L.adapt = g->adapt; L.q1 = g->q1; L.isym = g->isym; L.chg_ier = 0;
  }

  // P2 needs the unorm flag of iteration 0, set before the launch.
  Rec r = read_rec(rec);
  const int need_u0 = r.need_unorm;
  double pd = 0.0, pt = 0.0, pu = 0.0;
  // P0: scal part 1 -- u' = u*sqrt(d), w = 1/sqrt(d), rhs' = rhs*w.
  for (int s = s0 + warp; s < s1; s += nwarps) {
    int i = s * kSlice + lane;
    if (i < n) {
      double work = sqrt(a.diag[i]);
      a.u[i] = a.u[i] * work;
      double wv = 1.0 / work;
      a.w[i] = wv;
      a.rhs[i] = a.rhs[i] * wv;
      a.u1[i] = 0.0;
    }
  }
  if (!phase_sync(a, scalar_block, gen)) return;

  // P1: scaled off-diagonals, the reference's unscal drift of the resident
  // matrix, and the initial pseudo-residual d0 = pjac(u') + rhs' - u'.
  for (int s = s0 + warp; s < s1; s += nwarps) {
    int i = s * kSlice + lane;
    if (i < n) {
      int len = a.rlen[i];
      int base = a.sl_ptr[s] + lane;
      double wi = a.w[i];
      double ui = a.u[i];
      double winv_i = 1.0 / wi;
      double acc = a.rhs[i];
      for (int c0 = 0; c0 < len; c0 += kCh) {
        int jj[kCh];
        double vo[kCh], wj[kCh], uj[kCh];
#pragma unroll
        for (int k = 0; k < kCh; ++k)
          if (c0 + k < len) {
            int idx = base + (c0 + k) * kSlice;
            jj[k] = a.col[idx];
            vo[k] = a.offd[idx];
          }
#pragma unroll
        for (int k = 0; k < kCh; ++k)
          if (c0 + k < len) {
            wj[k] = a.w[jj[k]];
            uj[k] = a.u[jj[k]];
          }
#pragma unroll
        for (int k = 0; k < kCh; ++k)
          if (c0 + k < len) {
            int idx = base + (c0 + k) * kSlice;
            double sv = vo[k] * wi * wj[k];
            a.soff[idx] = sv;
            if (!a.defer_drift) a.offd[idx] = sv * winv_i * (1.0 / wj[k]);
            acc = acc - sv * uj[k];
          }
      }
      st_p4(p0 + i, 0.0, acc - ui, 0.0, 0.0);   // (dtwd0 later, d0, d(-1) = 0)
      a.diag[i] = winv_i * winv_i;
    }
  }
  if (!phase_sync(a, scalar_block, gen)) return;

  // P2: dtwd0 = -A' d0 and the iteration-0 norms; the scalar block runs
  // chgcon for in = 0 (ip = 0: cme = 0) while the rows work.
  {
    for (int s = s0 + warp; s < s1; s += nwarps) {
      int i = s * kSlice + lane;
      if (i < n) {
        int len = a.rlen[i];
        int base = a.sl_ptr[s] + lane;
        double acc = 0.0;
        for (int c0 = 0; c0 < len; c0 += kCh) {
          int jj[kCh];
          double vv[kCh], xx[kCh];
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) {
              int idx = base + (c0 + k) * kSlice;
              jj[k] = a.col[idx];
              vv[k] = a.soff[idx];
            }
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) xx[k] = p0[jj[k]].y;
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) acc = acc - vv[k] * xx[k];
        }
        p0[i].x = acc;
        double di = p0[i].y;
        pd += di * di;
        pt += di * acc;
        if (need_u0) { double ui = a.u[i]; pu += ui * ui; }
      }
    }
  }
  {
    if (scalar_block && threadIdx.x == 0 && L.adapt) chgcon_d(&L, t1, t2, 0);
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
  double *U[2] = {a.u, a.u1};
  for (int in = 0; in < a.itmax; ++in) {
    r = s_rec;
    if (r.halt) break;
    const double c1 = r.c1, c2 = r.c2, c3 = r.c3, c4 = r.c4;
    const int need_u = r.need_unorm;
    const P4 *pc = P[in % 2];
    P4 *pn = P[(in + 1) % 2];
    const double *uc = U[in % 2];
    double *un = U[(in + 1) % 2];
    double pd = 0.0, pt = 0.0, pu = 0.0;
    for (int s = s0 + warp; s < s1; s += nwarps) {
      int i = s * kSlice + lane;
      const int sn = s + nwarps;
      if (sn < s1)
        prefetch_slice(lane, a.sl_ptr[sn], a.sl_w[sn], sn * kSlice, a.col, a.soff, pc, uc, un);
      if (i < n) {
        const P4 me = ld_p4(pc + i);
        double unew = c1 * me.y + c2 * uc[i] + c3 * un[i];
        double dnew = c1 * me.x + c4 * me.y + c3 * me.z;
        int len = a.rlen[i];
        int base = a.sl_ptr[s] + lane;
        double acc = 0.0;
        for (int c0 = 0; c0 < len; c0 += kCh) {
          int jj[kCh];
          double vv[kCh];
          P4 xx[kCh];
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) {
              int idx = base + (c0 + k) * kSlice;
              jj[k] = a.col[idx];
              vv[k] = a.soff[idx];
            }
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) xx[k] = ld_p4(pc + jj[k]);
#pragma unroll
          for (int k = 0; k < kCh; ++k)
            if (c0 + k < len) {
              double dj = c1 * xx[k].x + c4 * xx[k].y + c3 * xx[k].z;
              acc = acc - vv[k] * dj;
            }
        }
        un[i] = unew;
        st_p4(pn + i, acc, dnew, me.y, 0.0);
        pd += dnew * dnew;
        pt += dnew * acc;
        if (need_u) pu += unew * unew;
      }
    }
    const int m = in + 1;
    if (scalar_block && threadIdx.x == 0 && L.adapt) chgcon_d(&L, t1, t2, m);
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
  r = s_rec;
  const int fin = r.in;
  const double *usol = U[fin % 2];

  // Optional peror (itpackv.F:607-720): the norms behind digit1/digit2.
  // pmult (itpackv.F:1970-2005) forms c = u - sum_j coef(:,j) u(jcoef).
  if (a.do_peror) {
    double pb = 0.0, pr = 0.0;
    for (int s = s0 + warp; s < s1; s += nwarps) {
      int i = s * kSlice + lane;
      if (i < n) {
        double wv = a.w[i];
        double wk = a.rhs[i] / wv;
        pb += wk * wk;
        int len = a.rlen[i];
        int base = a.sl_ptr[s] + lane;
        double cc = usol[i];
        for (int k = 0; k < len; ++k) {
          int idx = base + k * kSlice;
          cc = cc - a.soff[idx] * usol[a.col[idx]];
        }
        double wk2 = (a.rhs[i] - cc) / wv;
        pr += wk2 * wk2;
      }
    }
    bool ok = phase_reduce(a, scalar_block, gen, pb, pr, 0.0, 0.0,
                           [&](double sb, double sr, double, double) {
      if (scalar_block) {
        a.itp->dtnrm = sb;
        a.itp->unorm = sr;
      }
    });
    if (!ok) return;
  }

  // Epilogue: unscal (itpackv.F:2447-2477) and the GWCE eta update
  // (gwce.F:2006-2008).
  for (int s = s0 + warp; s < s1; s += nwarps) {
    int i = s * kSlice + lane;
    if (i < n) {
      double wv = a.w[i];
      double uf = usol[i] * wv;
      a.u[i] = uf;
      a.rhs[i] = a.rhs[i] * (1.0 / wv);
      if (a.eta_update) a.eta2[i] = a.nodecode[i] * (uf + 0.0) + a.eta1[i];
    }
  }
  if (scalar_block && threadIdx.x == 0) {
    int h = r.halt;
    if (h == 2) L.rparm1 = L.stptst;   // itpackv.F:394
    volatile Itp *g = a.itp;
    g->zeta = L.zeta; g->cme = L.cme; g->gamma = L.gamma; g->rho = L.rho;
    g->gamold = L.gamold; g->rhoold = L.rhoold; g->delnnm = L.delnnm; g->delsnm = L.delsnm;
    g->udnm = L.udnm; g->stptst = L.stptst; g->cmold = L.cmold; g->rparm1 = L.rparm1;
    g->adapt = L.adapt; g->q1 = L.q1; g->chg_ier = L.chg_ier;
    g->in = fin;
    g->halt = h;
    if (a.est) a.est->exact = 1;
    if (a.defer_drift == 1) *a.drift_pending = 1;
    a.flags->numitr = fin;
    a.flags->ier = (h == 2) ? 13 : 0;
    a.flags->zeta = L.rparm1;
    a.flags->cme = L.cme;
  }
}

// Per-solve ITPACK initialisation (echall, itpackv.F:1212-1255, plus the
// zeta floor of jcg :223-232); q1 and rparm1 persist across solves.
__global__ void jcg_clear_lines(unsigned long long *lines, int nwords) {
  griddep_wait();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nwords; k += gridDim.x * blockDim.x)
    lines[k] = kEmpty;
}

__global__ void jcg_init_kernel(Itp *it, Bar *bar, int itmax) {
  griddep_wait();
  bar->count = 0;
  it->zeta = it->rparm1;
  // cme keeps rparm(2) of the previous solve; chgcon(0) resets it to 0
  it->sme = -1.0;
  it->itmax = itmax;
  it->adapt = 1;
  it->isym = 0;
  it->in = 0;
  it->halt = 0;
  it->delnnm = it->delsnm = it->gamma = it->rho = it->stptst = it->udnm = 0.0;
  double temp = 512.0 * DBL_EPSILON;
  if (it->zeta < temp) it->zeta = temp;
  it->rec.halt = 0;
  it->rec.in = 0;
  it->rec.need_unorm = !it->q1;
}

}  // namespace adc

using namespace adc;

namespace adc {

// The dynamic shared memory a kernel may use is a per-function limit that
// every context in the process shares, so it is set to the most the device
// allows (its opt-in maximum less the kernel's static shared memory), not to
// one context's need: contexts with different layouts (the members of an
// ensemble) then all launch.
//
// The limit is also what a launch may ask for (`limit`).  It belongs to the
// device's context, which a host program may reset, so it is set for every
// layout.
int jcg_smem_limit(const void *fn, size_t *limit) {
  int dev = 0, optin = 0;
  ADC_CUDA(cudaGetDevice(&dev));
  ADC_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  ADC_CUDA(cudaFuncGetAttributes(&fa, fn));
  const size_t bytes = (size_t)optin - fa.sharedSizeBytes;
  ADC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  if (limit) *limit = bytes;
  return ADC_OK;
}

// Launch shape of the solver.  With host copies of the sliced ELL the
// resident kernel is planned first (not in the modes with FP32 parts), then
// the ordered one; without them, or where neither applies, jcg_kernel with as
// many 256-thread row blocks as can be co-resident (2 per SM), plus the scalar
// block.  A step of an FP64 shelf takes 637 us at 620k nodes (resident), 746
// at 660k and 1,137 at 800k (ordered; 1,190 and 1,373 with jcg_kernel), 1,523
// at 1,000k (ordered; 1,676), 1,786 at 1,061k (jcg_kernel).
int jcg_setup_grid(adc_ctx *c, const JcgHostSell *h) {
  int dev = 0, nsm = 0;
  ADC_CUDA(cudaGetDevice(&dev));
  ADC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  if (2 * sizeof(double) * (c->itmax + 1) > 48 * 1024) {
    set_error("itmax too large for the JCG scalar block");
    return ADC_ERR_ARG;
  }
  c->jcg_res = 0;
  if (h) {
    bool done = false;
    if (!any_f32(c))
      if (int rc = plan_jcg_resident(c, h, nsm, done)) return rc;
    if (!done)
      if (int rc = plan_jcg_ordered(c, h, nsm, done)) return rc;
    if (done) return ADC_OK;
  }
  // keep at least ~8 slices per block so the barrier cost stays amortised
  int nrb0 = std::max(1, std::min(2 * nsm - 1, std::max(1, c->nslices / 8)));
  if (c->jcg_nrb_req > 0) nrb0 = std::max(1, std::min({c->jcg_nrb_req, 2 * nsm - 1, c->nslices}));
  const void *fn = (const void *)jcg_kernel;
  size_t smem = 2 * sizeof(double) * (c->itmax + 1);
  if (int rc = jcg_smem_limit(fn)) return rc;
  int per_sm = 0;
  ADC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, smem));
  if (per_sm < 1) {
    set_error("jcg kernel cannot be resident");
    return ADC_ERR_CUDA;
  }
  const long long maxb = (long long)per_sm * nsm;
  const int nrb = (int)std::max<long long>(1, std::min<long long>(nrb0, maxb - 1));
  c->jcg_rows_blocks = nrb;
  c->jcg_grid = nrb + 1;
  c->jcg_smem = smem;
  return ADC_OK;
}

// Empties the barrier lines: before every solve of jcg_kernel, and once for
// newly allocated lines of the resident and the ordered kernel, whose
// generations then go on from solve to solve.
void jcg_clear_barrier(adc_ctx *c) {
  const int nwords = (int)(2 * 128 * (size_t)c->jcg_rows_blocks / 8);
  launch_k(jcg_clear_lines, 8, 256, c->stream, (unsigned long long *)c->jlines, nwords);
  c->launches++;
}

// Empties all that the solver's blocks have exchanged: for a new layout, and
// after a solve that gave up, which leaves posts of generations that the next
// solve would take for its own.
int jcg_reset_exchange(adc_ctx *c) {
  jcg_clear_barrier(c);
  const size_t bytes = (size_t)c->nslices * kSlice * sizeof(double4);
  ADC_CUDA(cudaMemsetAsync(c->jp[0], 0, bytes, c->stream));
  ADC_CUDA(cudaMemsetAsync(c->jp[1], 0, bytes, c->stream));
  ADC_CUDA(cudaStreamSynchronize(c->stream));
  return ADC_OK;
}

// What the last solve left undone of its estimate (have = false: nothing):
// chgcon over the recorded coefficients, some 10 us for a solve of 20
// iterations.  `head` and `pairs` are what the caller has copied of them
// already.
int jcg_estimate(const EstRec *est, cudaStream_t stream, Estimate &out, bool &have, const EstRec *head,
                 const double2 *pairs, int npairs) {
  have = false;
  EstRec r;
  if (head) {
    r = *head;
  } else {
    ADC_CUDA(cudaMemcpyAsync(&r, est, sizeof(r), cudaMemcpyDeviceToHost, stream));
    ADC_CUDA(cudaStreamSynchronize(stream));
  }
  if (r.exact || r.m < 0 || r.m > r.itmax) return ADC_OK;
  std::vector<double2> all;
  if (npairs < r.m) {
    all.resize(r.m);
    ADC_CUDA(cudaMemcpyAsync(all.data(), est + 1, r.m * sizeof(double2), cudaMemcpyDeviceToHost, stream));
    ADC_CUDA(cudaStreamSynchronize(stream));
    pairs = all.data();
  }
  std::vector<double> t1(r.m + 2), t2(r.m + 2);
  ItpLocal L;
  memset(&L, 0, sizeof(L));
  L.zeta = r.zeta;
  L.cme = r.cme0;
  L.cmold = r.cmold0;
  L.itmax = r.itmax;
  L.adapt = r.adapt0;
  for (int in = 0; in <= r.m && L.adapt; ++in) {
    if (in > 0) {
      L.gamma = pairs[in - 1].x;
      L.rho = pairs[in - 1].y;
    }
    if (in > 1) {
      L.gamold = pairs[in - 2].x;
      L.rhoold = pairs[in - 2].y;
    }
    chgcon_d(&L, t1.data(), t2.data(), in);
  }
  out.serial = r.serial;
  out.cme = L.cme;
  out.cmold = L.cmold;
  out.adapt = L.adapt;
  out.ier = L.chg_ier;
  out.stptst = L.cme != 1.0 ? r.sqd / (r.squd * (1.0 - L.cme)) : 1.0 / r.squd;   // pstop's tl / tr
  have = true;
  return ADC_OK;
}

// The step's flags, with the estimate of the last solve.
int read_state(adc_ctx *c, Flags &f, Estimate &est, bool &have) {
  constexpr int kPairs = 64;   // of most solves; more are copied apart
  struct {
    Flags f;
    char words[kEstOffset - sizeof(Flags)];
    EstRec r;
    double2 pairs[kPairs];
  } b;
  const int n = std::min(kPairs, c->itmax + 2);
  ADC_CUDA(cudaMemcpyAsync(&b, c->flags, kEstOffset + sizeof(EstRec) + n * sizeof(double2), cudaMemcpyDeviceToHost,
                           c->stream));
  ADC_CUDA(cudaStreamSynchronize(c->stream));
  f = b.f;
  est = c->est_last;
  have = !b.r.exact && est.serial == b.r.serial;
  if (!have) {
    if (int rc = jcg_estimate(c->est, c->stream, est, have, &b.r, b.pairs, n)) return rc;
    if (have) c->est_last = est;
  }
  if (have) f.cme = est.cme;
  return ADC_OK;
}

int launch_jcg_impl(adc_ctx *c, int eta_update, int do_peror, int run_init, int defer_drift, int d1) {
  JcgArgs a;
  a.do_peror = do_peror;
  a.n = c->np;
  a.nslices = c->nslices;
  a.nrb = c->jcg_rows_blocks;
  a.itmax = c->itmax;
  a.sl_ptr = c->sl_ptr;
  a.sl_w = c->sl_w;
  a.col = c->col;
  a.rlen = c->rlen;
  a.offd = c->offd;
  a.soff = c->soff;
  a.soff32 = c->soff32;
  a.diag = c->diag;
  a.rhs = c->gwce_lv;
  a.u = c->etas;
  a.u1 = c->ju1;
  a.p0 = c->jp[0];
  a.p1 = c->jp[1];
  a.w = c->jw;
  a.itp = c->itp;
  a.bar = c->bar;
  a.arrive = c->jlines;
  a.flags = c->flags;
  a.est = c->est;
  a.spin = c->spin_cycles > 0 ? c->spin_cycles : kSpinCycles;
  a.spin_mask = a.spin < 1000000 ? 0 : 63;   // 64 polls may take 100,000 cycles
  a.eta_update = eta_update;
  a.d1 = d1;
  a.nodecode = c->nodecode;
  a.nnodecode = c->nnodecode;
  a.dp = c->dp;
  a.h0 = c->p.h0;
  a.eta1 = c->eta1;
  a.eta2 = c->eta2;
  a.run_init = run_init;
  a.defer_drift = defer_drift;
  // the word after the step flags (allocated only by the time-step context)
  a.drift_pending = defer_drift ? (int *)(c->flags + 1) + 1 : nullptr;
  if (c->jcg_res == 1 || c->jcg_res == 2) {
    if (int rc = launch_jcg_resident(a, c)) return rc;
    c->launches++;
    return do_peror ? launch_jcg_peror(a, c) : ADC_OK;
  }
  if (c->jcg_res == 3) {
    if (int rc = launch_jcg_ordered(a, c)) return rc;
    c->launches++;
    return do_peror ? launch_jcg_peror(a, c) : ADC_OK;
  }
  jcg_clear_barrier(c);
  if (run_init) {
    launch_k(jcg_init_kernel, 1, 1, c->stream, c->itp, c->bar, c->itmax);
    c->launches++;
  }
  void *args[] = {&a};
  ADC_CUDA(cudaLaunchCooperativeKernel((const void *)jcg_kernel, dim3(c->jcg_grid), dim3(kThreads), args,
                                       c->jcg_smem, c->stream));
  c->launches++;
  return ADC_OK;
}

// The time-step solve defers the COEF drift to the next GWCE.  `d1` (not
// jcg_kernel): D1 of the wet/dry pass after the elevation update.
int launch_jcg(adc_ctx *c, int eta_update, bool d1) {
  // a mode with FP32 parts keeps no bitwise COEF history, so the drift is dropped
  return launch_jcg_impl(c, eta_update, 0, 1, any_f32(c) ? 2 : 1, d1);
}

}  // namespace adc
