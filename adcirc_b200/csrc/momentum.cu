// momentum.cu -- Mom_Eqs_New_NC (momentum.F:166-1208): lumped explicit
// non-conservative 2DDI momentum with IBPV lateral stress and corrected
// area integration, land boundary codes 0-19 and the zero normal velocity
// gradient of code 40, Cartesian coordinates.
//
// Two kernels: an element kernel forms the six load-vector contributions
// (momentum.F:298-699); a node kernel gathers them in element order, forms
// the nodal load and the 2x2 LHS (:713-803), applies the velocity boundary
// condition of the node if it has one (:810-862), solves (:1128-1138) and
// writes the fluxes (:1179-1182).  Boundary nodes in ME2GW are distinct,
// so the boundary step is a per-node operation.
#include "step_bodies.cuh"

namespace adc {

// 1,024 threads an SM (64 registers; with 768 threads of 80 the surge mesh's
// launch takes 52 us instead of 46) in blocks of two warps, whose gathers and
// arithmetic overlap better than those of eight (47 us).
constexpr int kMomThreads = 64;

template <class R>
__global__ void __launch_bounds__(kMomThreads, 1024 / kMomThreads) k_mom_elem(adc_ctx c, int alpha) {
  griddep_wait();
  __shared__ R sh[kMomThreads / 32][32 * 6];
  const int e0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31);
  if (e0 < c.ne) warp_mom<R>(c, e0, sh[threadIdx.x >> 5], alpha != 0);
}

// 64 registers: 39 us on the surge mesh, 44 with the compiler's 74.
// With `log`, also the end of a step of adc_run: its iteration count and the
// step table's cursor, which this kernel does not read.
template <class R>
__global__ void __launch_bounds__(kThreads, 4) k_mom_node(adc_ctx c, int *log, int cap) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.np) node_mom<R>(c, i);
  if (log && i == 0) step_end(c, log, cap);
}

__global__ void k_mom_zng(adc_ctx c) {
  griddep_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) one_zng(c);
}

// `whole`: the wet/dry pass precedes in the same call and leaves ALPHAL to
// the element pass; `log`: adc_run's iteration log.
int launch_momentum(adc_ctx *c, bool whole, int *log) {
  const int alpha = whole && c->p.nolifa == 2;
  kmark(c, KS_MOM_ELEM, 0);
  if (f32_momentum(c)) {   // FP32 element terms and their gather
    launch_k(k_mom_elem<float>, nblk(c->ne, kMomThreads), kMomThreads, c->stream, *c, alpha);
    kmark(c, KS_MOM_ELEM, 1);
    kmark(c, KS_MOM_NODE, 0);
    launch_k(k_mom_node<float>, nblk(c->np), kThreads, c->stream, *c, log, c->numitr_cap);
  } else {
    launch_k(k_mom_elem<double>, nblk(c->ne, kMomThreads), kMomThreads, c->stream, *c, alpha);
    kmark(c, KS_MOM_ELEM, 1);
    kmark(c, KS_MOM_NODE, 0);
    launch_k(k_mom_node<double>, nblk(c->np), kThreads, c->stream, *c, log, c->numitr_cap);
  }
  if (c->n_zng > 0) {
    launch_k(k_mom_zng, 1, 32, c->stream, *c);
    c->launches++;
  }
  kmark(c, KS_MOM_NODE, 1);
  c->launches += 2;
  return ADC_OK;
}

template __global__ void k_mom_elem<double>(adc_ctx, int);
template __global__ void k_mom_elem<float>(adc_ctx, int);
template __global__ void k_mom_node<double>(adc_ctx, int *, int);
template __global__ void k_mom_node<float>(adc_ctx, int *, int);

}  // namespace adc
