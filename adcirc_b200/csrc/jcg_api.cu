// jcg_api.cu -- the ITPACK entry points jcg / dfault (itpackv.F:63, 1070)
// with the reference's argument list, running the device JCG kernel.
//
// The host part mirrors what jcg does before iterating: echall
// (itpackv.F:1212-1255), the zeta floor (:223-232), and the structural half
// of scal (:2281-2391: diagonal moved to column 1, negative rows negated,
// zero diagonal -> ier 401, empty jcoef slots -> the row itself).  The
// system is then staged once in HBM in sliced-ELL form and solved by the
// persistent kernel of jcg.cu, which performs the numerical scal/unscal,
// the iteration and peror; the scaled-then-unscaled coefficients are
// copied back as the reference leaves them.
#include "adc_internal.cuh"

#include <cfloat>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>
#include <algorithm>

namespace adc {
int jcg_setup_grid(adc_ctx *c, const JcgHostSell *h);
int launch_jcg_impl(adc_ctx *c, int eta_update, int do_peror, int run_init, int defer_drift, int d1);

// ITPACK state that survives between jcg calls: itjcg's SAVEd q1 flag.
static int g_q1 = 0;
int jcg_q1_get() { return g_q1; }
void jcg_q1_set(int v) { g_q1 = v; }

// One call's device memory: one allocation.  (A cudaMalloc takes 1 to 3 ms
// for each block of a megabyte or more, and so does its cudaFree; the 18
// arrays of a 90k-row system were 20 to 70 ms around a solve of 0.12 ms.)
struct Stage {
  adc_ctx c;
  unsigned char *base = nullptr;
  size_t used = 0;
  Stage() { memset((void *)&c, 0, sizeof(c)); }
  ~Stage() {
    if (c.stream) {
      cudaStreamSynchronize(c.stream);   // copies from this call's host arrays
      cudaStreamDestroy(c.stream);
    }
    if (c.jtab && c.jtab != c.jtab_room) cudaFree(c.jtab);
    if (base) cudaFree(base);
  }
  // Places `n` elements: first for the size alone, then in the allocation.
  template <class T>
  void place(T **d, size_t n) {
    used = (used + 255) & ~(size_t)255;
    if (base) *d = (T *)(base + used);
    used += std::max<size_t>(n, 1) * sizeof(T);
  }
};

// The scalars a solve reads and leaves, copied together.
struct SolveState {
  Itp it;
  Bar bar;
  Flags fl;
};

// SELL slots from COEF as the caller holds it (columns of n rows), and back.
__global__ void k_slots_from_ell(int nnz, const int *src, const double *ell, double *off) {
  griddep_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nnz) off[t] = src[t] >= 0 ? ell[src[t]] : 0.0;
}
__global__ void k_slots_to_ell(int nnz, const int *src, const double *off, double *ell) {
  griddep_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nnz && src[t] >= 0) ell[src[t]] = off[t];
}

static int jcg_solve(int n, int ndim, int maxnz, int *jcoef, double *coef, double *rhs,
                     double *u, int itmax, int *iparm, double *rparm, int &ier, int &in_out,
                     double &stptst, double &cme, double &bnrm, double &rnrm) {
  // sliced ELL of the slots that take part in pjac: every j >= 2 except the
  // empty ones (jcoef == i and coef == 0, i.e. 0*u(i) terms)
  const int nslices = (n + kSlice - 1) / kSlice;
  const size_t npad = (size_t)nslices * kSlice;
  std::vector<int> rlen(npad, 0), sl_w(nslices, 0), sl_ptr(nslices + 1, 0);
  for (int j = 1; j < maxnz; ++j) {
    const int *jc = jcoef + (size_t)ndim * j;
    const double *cf = coef + (size_t)ndim * j;
    for (int i = 0; i < n; ++i) rlen[i] += !(jc[i] == i + 1 && cf[i] == 0.0);
  }
  for (int i = 0; i < n; ++i) sl_w[i / kSlice] = std::max(sl_w[i / kSlice], rlen[i]);
  size_t rcol = 0;
  for (int s = 0; s < nslices; ++s) {
    sl_ptr[s + 1] = sl_ptr[s] + sl_w[s] * kSlice;
    rcol += 512 * ((sl_w[s] + 7) / 8);
  }
  const int nnz = sl_ptr[nslices];
  // column and source of each slot; both arrays are written in full
  const std::unique_ptr<int[]> col(new int[std::max(nnz, 1)]), src(new int[std::max(nnz, 1)]);
  for (int s = 0; s < nslices; ++s) {
    int at[kSlice] = {0};
    const int i0 = s * kSlice, lanes = std::min(kSlice, n - i0);
    int *cs = col.get() + sl_ptr[s], *ss = src.get() + sl_ptr[s];
    for (int j = 1; j < maxnz; ++j)
      for (int l = 0; l < lanes; ++l) {
        const size_t k = i0 + l + (size_t)ndim * j;
        if (jcoef[k] == i0 + l + 1 && coef[k] == 0.0) continue;
        const int q = at[l]++ * kSlice + l;
        cs[q] = jcoef[k] - 1;
        ss[q] = i0 + l + n * j;
      }
    for (int l = 0; l < kSlice; ++l)
      for (int q = at[l] * kSlice + l; q < sl_w[s] * kSlice; q += kSlice) {
        cs[q] = l < lanes ? i0 + l : 0;
        ss[q] = -1;
      }
  }
  Stage st;
  adc_ctx &c = st.c;
  c.np = n;
  c.nslices = nslices;
  c.nnz_pad = nnz;
  c.itmax = itmax;
  if (cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking) != cudaSuccess) return ADC_ERR_CUDA;
  double *d_ell = nullptr;
  int *d_src = nullptr;
  SolveState *d_state = nullptr;
  // room for the solver's tables: packed columns, and at most every slot a
  // halo node that some block sends
  const size_t room = rcol + 14 * (size_t)nnz + 4 * npad + (64u << 10);
  const size_t nlines = 2 * 128 * 1024;   // of up to 1,024 row blocks (two per SM at most)
  size_t zero0 = 0;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) ADC_CUDA(cudaMalloc((void **)&st.base, st.used));
    st.used = 0;
    st.place(&c.sl_ptr, nslices + 1);
    st.place(&c.sl_w, nslices);
    st.place(&c.col, nnz);
    st.place(&c.rlen, npad);
    st.place(&c.offd, nnz);
    st.place(&c.soff, nnz);
    st.place(&c.diag, n);
    st.place(&c.gwce_lv, n);
    st.place(&d_ell, (size_t)n * maxnz);
    st.place(&d_src, nnz);
    st.place(&d_state, 1);
    st.place((char **)&c.est, sizeof(EstRec) + (itmax + 2) * sizeof(double2));
    st.place(&c.jtab_room, room);
    st.place((char **)&c.jlines, nlines);
    zero0 = (st.used + 255) & ~(size_t)255;   // from here on zeroed
    st.place(&c.etas, npad);
    st.place(&c.ju1, npad);
    st.place(&c.jw, npad);
    st.place(&c.jp[0], npad);
    st.place(&c.jp[1], npad);
  }
  c.jtab_cap = room;
  c.itp = &d_state->it;
  c.bar = &d_state->bar;
  c.flags = &d_state->fl;
  // everything in stream order (pageable copies may still be on their way
  // when the call returns)
  auto up = [&](void *d, const void *h, size_t bytes) {
    return bytes ? cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, c.stream) : cudaSuccess;
  };
  ADC_CUDA(cudaMemsetAsync(st.base + zero0, 0, st.used - zero0, c.stream));
  ADC_CUDA(up(c.sl_ptr, sl_ptr.data(), sl_ptr.size() * sizeof(int)));
  ADC_CUDA(up(c.sl_w, sl_w.data(), sl_w.size() * sizeof(int)));
  ADC_CUDA(up(c.col, col.get(), (size_t)nnz * sizeof(int)));
  ADC_CUDA(up(c.rlen, rlen.data(), rlen.size() * sizeof(int)));
  ADC_CUDA(up(d_src, src.get(), (size_t)nnz * sizeof(int)));
  ADC_CUDA(up(c.diag, coef, n * sizeof(double)));
  ADC_CUDA(up(c.gwce_lv, rhs, n * sizeof(double)));
  ADC_CUDA(up(c.etas, u, n * sizeof(double)));
  ADC_CUDA(cudaMemcpy2DAsync(d_ell, n * sizeof(double), coef, (size_t)ndim * sizeof(double), n * sizeof(double),
                             maxnz, cudaMemcpyHostToDevice, c.stream));
  launch_k(k_slots_from_ell, std::max(1, nblk(nnz)), kThreads, c.stream, nnz, (const int *)d_src,
           (const double *)d_ell, c.offd);
  const JcgHostSell hs{sl_ptr.data(), sl_w.data(), col.get(), rlen.data()};
  int rc = jcg_setup_grid(&c, &hs);
  if (rc) return rc;
  if (2 * 128 * (size_t)c.jcg_rows_blocks > nlines) { set_error("JCG barrier lines"); return ADC_ERR_ARG; }
  jcg_clear_barrier(&c);
  SolveState ss;
  memset((void *)&ss, 0, sizeof(ss));
  Itp &it = ss.it;
  it.zeta = rparm[0];
  it.rparm1 = rparm[0];
  it.cme = rparm[1];
  it.sme = (rparm[2] == 0.0) ? -1.0 : rparm[2];
  it.itmax = itmax;
  it.adapt = (iparm[5] == 1 || iparm[5] == 3) ? 1 : 0;
  it.q1 = g_q1;
  it.srelpr = DBL_EPSILON;
  double temp = 512.0 * DBL_EPSILON;
  if (it.zeta < temp) it.zeta = temp;
  it.rec.need_unorm = !it.q1;
  ADC_CUDA(up(d_state, &ss, sizeof(ss)));
  EstRec er;
  memset((void *)&er, 0, sizeof(er));
  er.exact = 1;   // what a kernel other than the resident one leaves
  ADC_CUDA(up(c.est, &er, sizeof(er)));
  rc = launch_jcg_impl(&c, 0, iparm[11] >= 0 ? 1 : 0, 0, 0, 0);
  if (rc) return rc;
  launch_k(k_slots_to_ell, std::max(1, nblk(nnz)), kThreads, c.stream, nnz, (const int *)d_src,
           (const double *)c.offd, d_ell);
  ADC_CUDA(cudaMemcpyAsync(&ss, d_state, sizeof(ss), cudaMemcpyDeviceToHost, c.stream));
  ADC_CUDA(cudaStreamSynchronize(c.stream));
  const Flags &fl = ss.fl;
  if (fl.timeout) { set_error("JCG barrier wait expired"); return ADC_ERR_TIMEOUT; }
  auto down = [&](void *h, const void *d, size_t bytes) {
    return cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, c.stream);
  };
  ADC_CUDA(down(u, c.etas, n * sizeof(double)));
  ADC_CUDA(down(rhs, c.gwce_lv, n * sizeof(double)));
  ADC_CUDA(down(coef, c.diag, n * sizeof(double)));
  if (maxnz > 1)
    ADC_CUDA(cudaMemcpy2DAsync(coef + ndim, (size_t)ndim * sizeof(double), d_ell + n, n * sizeof(double),
                               n * sizeof(double), maxnz - 1, cudaMemcpyDeviceToHost, c.stream));
  Estimate est;
  bool have;
  if (int rc2 = jcg_estimate(c.est, c.stream, est, have)) return rc2;   // waits for the copies above
  if (have) {
    it.cme = est.cme;
    it.stptst = est.stptst;
  }
  g_q1 = it.q1;
  ier = fl.ier;
  in_out = it.in;
  stptst = it.stptst;
  cme = it.cme;
  bnrm = it.dtnrm;
  rnrm = it.unorm;
  return ADC_OK;
}

}  // namespace adc

using namespace adc;

extern "C" {

void adc_dfault(int *iparm, double *rparm) {
  // dfault, itpackv.F:1070-1170 (srelpr = 2**-52 for IEEE double)
  const double srelpr = DBL_EPSILON;
  const int ip[12] = {100, -1, 0, 6, 0, 1, 1, 0, -2, 0, 0, 3};
  for (int k = 0; k < 12; ++k) iparm[k] = ip[k];
  rparm[0] = 5.0e-6; rparm[1] = 0.0; rparm[2] = 0.0; rparm[3] = 0.75; rparm[4] = 1.0;
  rparm[5] = 0.0; rparm[6] = 0.25; rparm[7] = 128.0 * srelpr; rparm[8] = 0.0;
  rparm[9] = 0.0; rparm[10] = 0.0; rparm[11] = 0.0;
}

void adc_jcg_reset(void) { g_q1 = 0; }

void adc_jcg(const int *n_, const int *ndim_, const int *maxnz_, int *jcoef, double *coef,
             double *rhs, double *u, int *iwksp, const int *nw_, double *wksp, int *iparm,
             double *rparm, int *ier) {
  (void)iwksp;
  (void)wksp;
  *ier = 0;
  const int n = *n_, ndim = *ndim_, maxnz = *maxnz_, nw = *nw_;
  if (iparm[0] <= 0) return;
  const int itmax = iparm[0];
  if (n <= 0) { *ier = 11; return; }
  if (ndim < n || maxnz < 1) { *ier = 11; set_error("ndim < n or maxnz < 1"); return; }
  // structural part of scal (itpackv.F:2340-2391)
  int nsgncg = 0;
  for (int i = 1; i <= n; ++i) {
    int *jr = jcoef + (i - 1);
    double *cr = coef + (i - 1);
    if (jr[0] != i) {
      if (maxnz < 2) { *ier = 402; return; }
      for (int j = 2; j <= maxnz; ++j) {
        size_t k = (size_t)ndim * (j - 1);
        if (jr[k] == i) {
          double save = cr[k];
          cr[k] = cr[0];
          jr[k] = jr[0];
          cr[0] = save;
          jr[0] = i;
        }
      }
    }
    if (cr[0] < 0.0) {
      for (int j = 1; j <= maxnz; ++j) cr[(size_t)ndim * (j - 1)] = -cr[(size_t)ndim * (j - 1)];
      rhs[i - 1] = -rhs[i - 1];
      nsgncg++;
    } else if (cr[0] == 0.0) {
      *ier = 401;
      return;
    }
  }
  for (int j = 2; j <= maxnz; ++j)
    for (int i = 1; i <= n; ++i)
      if (jcoef[(i - 1) + (size_t)ndim * (j - 1)] <= 0) jcoef[(i - 1) + (size_t)ndim * (j - 1)] = i;
  auto restore_zeros = [&]() {
    for (int j = 2; j <= maxnz; ++j)
      for (int i = 1; i <= n; ++i)
        if (jcoef[(i - 1) + (size_t)ndim * (j - 1)] == i) jcoef[(i - 1) + (size_t)ndim * (j - 1)] = 0;
  };
  if (nsgncg > 0 && nsgncg < n) {
    // ITPACK would switch to the nonsymmetric eigenvalue routine
    // (isym = 1, eigvns/eqrt1s); that branch is not implemented.
    *ier = 903;
    restore_zeros();
    set_error("mixed-sign diagonal (ITPACK isym branch) not supported");
    return;
  }
  iparm[7] = 4 * n + 4 * itmax;
  if (nw < iparm[7]) {
    *ier = 12;
    restore_zeros();
    return;
  }
  int e = 0, in = 0;
  double stptst = 0, cme = 0, bnrm = 0, rnrm = 0;
  int rc = jcg_solve(n, ndim, maxnz, jcoef, coef, rhs, u, itmax, iparm, rparm, e, in, stptst,
                     cme, bnrm, rnrm);
  if (rc != ADC_OK) {
    *ier = 904;
    restore_zeros();
    return;
  }
  restore_zeros();
  *ier = e;
  if (e == 13 && iparm[2] == 0) rparm[0] = stptst;
  double digit1 = rparm[10], digit2 = rparm[11];
  if (iparm[11] >= 0) {
    const double srelpr = DBL_EPSILON;
    digit1 = -std::log10(std::fabs(srelpr));
    if (stptst > 0.0) digit1 = -std::log10(std::fabs(stptst));
    if (bnrm == 0.0) {
      digit2 = -std::log10(std::fabs(srelpr));
    } else {
      double temp = rnrm / bnrm;
      digit2 = (temp == 0.0) ? -std::log10(std::fabs(srelpr)) : -std::log10(std::fabs(temp)) / 2.0;
    }
  }
  iparm[7] = iparm[7] - 4 * (itmax - in);
  if (iparm[2] != 0) return;
  iparm[0] = in;
  rparm[1] = cme;
  rparm[2] = (rparm[2] == 0.0) ? -1.0 : rparm[2];
  rparm[10] = digit1;
  rparm[11] = digit2;
}

}  // extern "C"
