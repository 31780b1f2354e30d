// sync.cu -- the state on its way to the bound host arrays (adc_sync_to_host).
//
// What bounds it is the copies, not the data.  A copy into pageable memory
// costs 10 to 12 us and moves 17 GB/s, and there are 31 arrays: 0.37 ms of a
// 651-node mesh's 0.2 MB.  So a state of up to 4 MB goes through the two
// halves of a pinned block: a kernel packs the next piece into one at PCIe
// speed while the host puts the last one's arrays in their places (0.1 ms per
// MB: beyond some 6 MB the direct copies are the faster way).  COEF is laid
// out as the reference holds it, COEF(NP,MNEI), on the device: the host's
// loop over the slots took 15 of the 28 ms of a 600k-node mesh.  A sync takes
// 0.45 -> 0.1 ms at 651 nodes, 9.6 -> 4.6 ms at 250k, 28 -> 13 ms at 600k.
#include <vector>

#include "step_bodies.cuh"

namespace adc {

__global__ void k_lhs_drift(adc_ctx c);
__global__ void k_lhs_drift_done(adc_ctx c);

// COEF's entry e = i + NP*j: the diagonal, the row's slots, zeros.
__device__ __forceinline__ double coef_entry(const adc_ctx &c, size_t e) {
  const int j = (int)(e / c.np), i = (int)(e - (size_t)j * c.np);
  if (j == 0) return c.diag[i];
  if (j > c.rlen[i]) return 0.0;
  return c.offd[c.sl_ptr[i / kSlice] + (j - 1) * kSlice + i % kSlice];
}

// Entries [e0, e0 + n) of COEF.
__global__ void k_coef_entries(adc_ctx c, size_t e0, size_t n, double *out) {
  griddep_wait();
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t < n) out[t] = coef_entry(c, e0 + t);
}

constexpr int kPackMax = 34;

struct PackTable {
  int n;
  const void *src[kPackMax];       // null: COEF
  unsigned first[kPackMax + 1];    // first 8-byte word in the block
  unsigned count[kPackMax];        // elements
  unsigned is_int;                 // bit per array: 4-byte elements, two to a word
  unsigned is_int_hi;              // (arrays 32 and up)
};

__device__ __forceinline__ bool seg_int(const PackTable &t, int s) {
  return (s < 32 ? t.is_int >> s : t.is_int_hi >> (s - 32)) & 1;
}

// Words [w0, w0 + n) of the packed state.
__global__ void k_pack(adc_ctx c, PackTable t, unsigned w0, unsigned n, unsigned long long *out) {
  griddep_wait();
  const unsigned o = blockIdx.x * blockDim.x + threadIdx.x, w = w0 + o;
  if (o >= n) return;
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int m = (lo + hi + 1) >> 1;
    if (t.first[m] <= w) lo = m; else hi = m - 1;
  }
  const unsigned k = w - t.first[lo];
  unsigned long long v;
  if (!t.src[lo]) {
    v = __double_as_longlong(coef_entry(c, k));
  } else if (seg_int(t, lo)) {
    const unsigned *p = (const unsigned *)t.src[lo];
    v = p[2 * k];
    if (2 * k + 1 < t.count[lo]) v |= (unsigned long long)p[2 * k + 1] << 32;
  } else {
    v = ((const unsigned long long *)t.src[lo])[k];
  }
  out[o] = v;
}

struct HostCopy {
  void *h;
  const void *d;    // null: COEF
  size_t n;
  int size;         // bytes per element
};

static std::vector<HostCopy> state_copies(const adc_ctx *c) {
  const adc_arrays_t *a = &c->host;
  const size_t np = c->np, ne = c->ne;
  std::vector<HostCopy> v = {
      {a->eta1, c->eta1, np, 8},           {a->eta2, c->eta2, np, 8},
      {a->etas, c->etas, np, 8},           {a->uu1, c->uu1, np, 8},
      {a->vv1, c->vv1, np, 8},             {a->uu2, c->uu2, np, 8},
      {a->vv2, c->vv2, np, 8},             {a->qx1, c->qx1, np, 8},
      {a->qy1, c->qy1, np, 8},             {a->qx2, c->qx2, np, 8},
      {a->qy2, c->qy2, np, 8},             {a->h1, c->h1, np, 8},
      {a->h2, c->h2, np, 8},               {a->tk, c->tk, np, 8},
      {a->tkm, c->tkm, 3 * np, 8},         {a->totalarea, c->totalarea, np, 8},
      {a->alphal, c->alphal, ne, 8},       {a->wsx1, c->wsx1, np, 8},
      {a->wsy1, c->wsy1, np, 8},           {a->wsx2, c->wsx2, np, 8},
      {a->wsy2, c->wsy2, np, 8},           {a->pr1, c->pr1, np, 8},
      {a->pr2, c->pr2, np, 8},             {a->gwce_lv, c->gwce_lv, np, 8},
      {a->mom_lv_x, c->mom_x, np, 8},      {a->mom_lv_y, c->mom_y, np, 8},
      {a->nodecode, c->nodecode, np, 4},   {a->nnodecode, c->nnodecode, np, 4},
      {a->noff, c->noff, ne, 4},           {a->mju, c->mju, np, 4},
      {a->coef, nullptr, np * c->mnei, 8}, {a->obccoef, c->obccoef, (size_t)c->neta * (c->mnei - 1), 8}};
  std::vector<HostCopy> w;
  for (const HostCopy &x : v)
    if (x.h && x.n) w.push_back(x);
  return w;
}

static size_t words_of(const HostCopy &x) { return (x.n * x.size + 7) / 8; }

constexpr size_t kPackBytes = 4u << 20;      // states that go packed
constexpr size_t kBlockBytes = 512u << 10;   // pinned: 0.6 ms of a bind; 1.6 MB took 2.2 ms

// The pinned block, if the state is small (at bind; the context keeps it).
void sync_setup(adc_ctx *c) {
  size_t words = 0;
  for (const HostCopy &x : state_copies(c)) words += words_of(x);
  c->h_pack = nullptr;
  if (words * 8 > kPackBytes) return;
  c->pack_half = std::min(words, kBlockBytes / 16);
  const size_t bytes = (words > c->pack_half ? 2 : 1) * c->pack_half * 8;
  if (cudaHostAlloc((void **)&c->h_pack, bytes, cudaHostAllocDefault) != cudaSuccess) {
    c->h_pack = nullptr;   // no pinned memory: array by array
    cudaGetLastError();
  }
}

// Words [w0, w0 + n) of the packed state to their arrays.
static void unpack(const std::vector<HostCopy> &v, const PackTable &t, size_t w0, size_t n,
                   const unsigned long long *from) {
  for (int s = 0; s < t.n; ++s) {
    const size_t a = std::max<size_t>(w0, t.first[s]), b = std::min<size_t>(w0 + n, t.first[s + 1]);
    if (a >= b) continue;
    const size_t o = (a - t.first[s]) * 8, end = std::min((b - t.first[s]) * 8, v[s].n * v[s].size);
    memcpy((char *)v[s].h + o, from + (a - w0), end - o);
  }
}

int download_state(adc_ctx *c) {
  const std::vector<HostCopy> v = state_copies(c);
  if (c->host.coef) {
    // COEF as the reference holds it: apply a drift the last solve left pending
    launch_k(k_lhs_drift, nblk(c->np), kThreads, c->stream, *c);
    launch_k(k_lhs_drift_done, 1, 1, c->stream, *c);
  }
  if (c->h_pack) {
    PackTable t;
    memset(&t, 0, sizeof(t));
    t.n = (int)v.size();
    for (int s = 0; s < t.n; ++s) {
      t.src[s] = v[s].d;
      t.count[s] = (unsigned)v[s].n;
      if (v[s].size == 4) (s < 32 ? t.is_int : t.is_int_hi) |= 1u << (s & 31);
      t.first[s + 1] = t.first[s] + (unsigned)words_of(v[s]);
    }
    const size_t words = t.first[t.n], half = c->pack_half;
    for (size_t w0 = 0, k = 0; w0 < words + half; w0 += half, ++k) {   // one piece ahead of the host
      if (w0 > 0) ADC_CUDA(cudaStreamSynchronize(c->stream));
      if (w0 < words) {
        const unsigned n = (unsigned)std::min(half, words - w0);
        launch_k(k_pack, nblk(n), kThreads, c->stream, *c, t, (unsigned)w0, n, c->h_pack + (k & 1) * half);
        ADC_CUDA(cudaGetLastError());
      }
      if (w0 > 0) unpack(v, t, w0 - half, std::min(half, words - (w0 - half)), c->h_pack + ((k - 1) & 1) * half);
    }
    return ADC_OK;
  }
  ADC_CUDA(cudaGetLastError());
  ADC_CUDA(cudaStreamSynchronize(c->stream));
  const size_t cap = 9 * (size_t)c->ne;   // doubles of the element scratch
  for (const HostCopy &x : v) {
    if (x.d) {
      ADC_CUDA(cudaMemcpy(x.h, x.d, x.n * x.size, cudaMemcpyDeviceToHost));
      continue;
    }
    for (size_t e0 = 0; e0 < x.n; e0 += cap) {
      const size_t n = std::min(cap, x.n - e0);
      launch_k(k_coef_entries, nblk(n), kThreads, c->stream, *c, e0, n, c->ebuf);
      ADC_CUDA(cudaGetLastError());
      ADC_CUDA(cudaStreamSynchronize(c->stream));
      ADC_CUDA(cudaMemcpy((double *)x.h + e0, c->ebuf, n * sizeof(double), cudaMemcpyDeviceToHost));
    }
  }
  return ADC_OK;
}

}  // namespace adc
