// wetdry.cu -- computeWettingAndDrying (wetdry.F:140-1470) and computeAlpha
// (wetdry.F:1561-1652): non-subgrid 2DDI, NDDT = 0, default NOFF rules.
// With internal barriers the nodes that receive overflow (NIBNODECODE, set
// by the flux step) wet their elements' nodes through NIBCNT (W2a/W2b,
// wetdry.F:813-816, 1086-1090) and exempt those elements from DE1 (:1114).
//
// Flags are integers and every pass except one is order independent, so
// node and element passes run one thread per item.  The exception is the
// W1 friction update (wetdry.F:593-618): it applies, in element order,
// TK(a) = TK(b) = max(candidate, TK(a), TK(b)) for each wetting event.
// Events are compacted per block in element order, and one block resolves
// the ordered list through each event's predecessors on its two nodes
// (block_chain, wd_chain.cuh), which reproduces the sequential result exactly.
#include "wd_chain.cuh"

namespace adc {

__global__ void k_wd_d1(adc_ctx c) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) c.flags->n_w1_events = 0;
  if (i < c.np) node_d1(c, i);
}

__global__ void __launch_bounds__(kW1Block) k_wd_w1(adc_ctx c) {
  griddep_wait();
  block_w1(c, blockIdx.x);
}

__global__ void __launch_bounds__(1024) k_wd_chain(adc_ctx c) {
  griddep_wait();
  block_chain(c);
}

__global__ void k_wd_w2b(adc_ctx c) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.np) node_w2b(c, i);
}

__global__ void k_wd_de1(adc_ctx c) {
  griddep_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < c.ne) elem_de1(c, e);
}

__global__ void k_wd_d2(adc_ctx c) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.np) node_d2(c, i);
}

__global__ void k_h2_update(adc_ctx c) {
  griddep_wait();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.np) return;
  c.h2[i] = c.dp[i] + c.p.ifnlfa * c.eta2[i];
}

__global__ void k_wd_alpha(adc_ctx c) {
  griddep_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < c.ne) c.alphal[e] = elem_alpha(c, e);
}

// `whole`: the momentum pass follows and forms ALPHAL; `d1_done`: the solve
// has done D1.
int launch_wetdry(adc_ctx *c, bool whole, bool d1_done) {
  const adc_ctx &cv = *c;
  if (c->p.nolifa != 2) {
    launch_k(k_h2_update, nblk(c->np), kThreads, c->stream, cv);
    c->launches++;
    return ADC_OK;
  }
  if (!d1_done) {
    launch_k(k_wd_d1, nblk(c->np), kThreads, c->stream, cv);
    c->launches++;
  }
  launch_k(k_wd_w1, c->ev_blocks, kW1Block, c->stream, cv);
  launch_k(k_wd_chain, 1, 1024, c->stream, cv);
  if (c->nfluxib) {
    launch_k(k_wd_w2b, nblk(c->np), kThreads, c->stream, cv);
    c->launches++;
  }
  launch_k(k_wd_de1, nblk(c->ne), kThreads, c->stream, cv);
  launch_k(k_wd_d2, nblk(c->np), kThreads, c->stream, cv);
  c->launches += 4;
  if (!whole) {
    launch_k(k_wd_alpha, nblk(c->ne), kThreads, c->stream, cv);
    c->launches++;
  }
  return ADC_OK;
}

}  // namespace adc
