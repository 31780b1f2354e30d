// jcg_common.cuh -- launch arguments of the three JCG kernels (jcg.cu,
// jcg_resident.cu, jcg_ordered.cu) and the host entry points of the two with
// block-local tables.
#pragma once

#include "adc_internal.cuh"

#include <cstring>
#include <vector>

namespace adc {

struct JcgArgs {
  int n, nslices, nrb, itmax;
  const int *sl_ptr, *sl_w, *col, *rlen;
  double *offd, *soff, *diag, *rhs;
  float *soff32;                // FP32 copy of the scaled matrix (mixed mode)
  double *u, *u1, *w;
  double4 *p0, *p1;
  Itp *itp;
  Bar *bar;
  void *arrive;             // the barrier lines (see the kernels)
  Flags *flags;
  EstRec *est;              // resident kernel: what the estimate's last value is formed from, if not here
  long long spin;           // cycles a wait may take ...
  unsigned spin_mask;       // ... and polls between looks at the clock and the timeout flag, less one
  int eta_update;
  int do_peror;
  int run_init;               // echall's per-solve initialisation inside the kernel
  int defer_drift;            // 1: leave the COEF unscal drift to the next step;
                              // 2: drop it (mixed mode, COEF is rebuilt or kept as is)
  int *drift_pending;         // set to 1 when the drift is left pending
  int d1;                     // the epilogue ends with wet/dry pass D1 (wetdry.F:234-285)
  int *nodecode, *nnodecode;
  const double *eta1, *dp;
  double *eta2;
  double h0;
  // jcg_ordered.cu: block-local 16-bit columns per slot, rows other blocks read
  const unsigned short *lcol;
  const unsigned char *exp;
  int stage_wcap;             // widest slice that is staged; wider ones are read in place
  // resident kernel (jcg_resident.cu); the sizes in jcg_ordered.cu too
  int rows_max;               // rows of the largest row block
  int halo_max;               // halo nodes of the largest row block
  int stage_bytes;            // one staged slice
  const int4 *meta;           // per slice: first slot, width, column words before it, resident offset
  const uint4 *rcol;          // block-local columns as byte offsets, 8 per lane and word
  const unsigned char *rle;   // per row: length, top bit: read by another row block
  const int *halo_ptr;        // [nrb + 1] into halo_ids
  const int *halo_ids;        // halo nodes of each row block
  const int *push_ptr;        // cluster form: [nrb + 1] into push
  const int2 *push;           // values a block sends: local row, (receiver << 16) | halo place
  int o_hp, o_hid, o_tri, o_meta, o_part, o_bar, o_push, o_area, o_res;   // shared-memory offsets
};

int launch_jcg_resident(const JcgArgs &a, const adc_ctx *c);
int plan_jcg_resident(adc_ctx *c, const JcgHostSell *h, int nsm, bool &done);
int launch_jcg_ordered(const JcgArgs &a, const adc_ctx *c);
int plan_jcg_ordered(adc_ctx *c, const JcgHostSell *h, int nsm, bool &done);
int jcg_smem_limit(const void *fn, size_t *limit = nullptr);

// A kernel's host tables, gathered for one allocation and one copy
// (adc_ctx::jtab).
struct JcgTables {
  std::vector<unsigned char> h;
  template <class T>
  size_t add(const std::vector<T> &v) {
    const size_t o = (h.size() + 255) & ~(size_t)255;
    h.resize(o + v.size() * sizeof(T));
    if (!v.empty()) memcpy(h.data() + o, v.data(), v.size() * sizeof(T));
    return o;
  }
  int upload(adc_ctx *c) const {
    if (h.size() + 256 <= c->jtab_cap) c->jtab = c->jtab_room;
    else ADC_CUDA(cudaMalloc((void **)&c->jtab, h.size() + 256));
    ADC_CUDA(cudaMemcpyAsync(c->jtab, h.data(), h.size(), cudaMemcpyHostToDevice, c->stream));
    ADC_CUDA(cudaStreamSynchronize(c->stream));
    return ADC_OK;
  }
};
int launch_jcg_peror(const JcgArgs &a, adc_ctx *c);

}  // namespace adc
