// gwce.cu -- GWCE_New (gwce.F:237-2111) for IM=0 (Kolar-Gray lateral
// stress, non-conservative advection), consistent mass (ILump = 0),
// Cartesian coordinates, plus the TIMESTEP glue that precedes it.
//
// Element terms are computed once per element into a scratch buffer and
// gathered per node over the node->element CSR in increasing element order,
// i.e. the order of the reference's scatter loops, starting from zero as
// the reference does after zeroing.  No atomics touch floating point, so
// the results are deterministic and, compiled without FMA contraction,
// reproduce the serial arithmetic bit for bit.
//
// Four passes: nodes (shift, friction, vortex forcing), elements (matrix
// entries or the pending drift, and load-vector terms), nodes (their
// gathers; the last block forms EP), boundary rows.  Separate kernels for
// the matrix and the load vector, and single-thread kernels between them,
// took eleven launches of 1.5 to 2 us each on meshes too small to fill the
// GPU, and two more passes over the elements' NM, NOFF and ALPHAL.  Measured
// with the folds into the solve and the momentum passes (23 launches a step to
// 13): 83 -> 76 us a step on the 533-node beach, 156 -> 143 us on a 25k-node
// shelf.
#include "step_bodies.cuh"

#include <algorithm>

namespace adc {

// The step's first pass.  Every block forms the storm's state itself; the
// last one to finish keeps it.
__global__ void __launch_bounds__(kThreads) k_step_begin(adc_ctx c, const adc_step_t *steps, int whole) {
  griddep_wait();
  __shared__ VortexState v;
  __shared__ int past;
  const adc_step_t st = steps[c.flags->cursor];
  if (c.vortex_on) {
    if (threadIdx.x == 0) {
      v = *c.vstate;
      past = vortex_advance(c, st.timeloc, v);
    }
  }
  // the other warps' shift hides the first thread's chain of divisions
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.np) node_shift(c, st, i, whole != 0, c.vortex_on != 0);
  if (c.vortex_on) {
    __syncthreads();
    if (i < c.np) node_vortex(c, v, st.rampmete, i);
  }
  // every block has read the old state before it takes its ticket
  if (c.vortex_on && threadIdx.x == 0 && atomicAdd(&c.tickets[0], 1) == (int)gridDim.x - 1) {
    c.tickets[0] = 0;
    *c.vstate = v;
    if (past) c.flags->status = ADC_ERR_ARG;
  }
}

// Met forcing supplied by the host for this step (WSX2, WSY2, PR2).
__global__ void k_apply_met(adc_ctx c) {
  griddep_wait();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.np) return;
  c.wsx2[i] = c.met_wsx[i];
  c.wsy2[i] = c.met_wsy[i];
  c.pr2[i] = c.met_pr[i];
}

// The step's LHS decision (gwce.F:430-431): rebuild when NCChange > 0, else
// apply a drift of COEF that the last solve left pending.  The words after
// the flags: [0] the decision, [1] drift pending, [2] drift applied, [3] the
// next rebuild gathers every row.  Decision and words change only in the last
// block of k_gwce_node, when every block has read them.
__device__ __forceinline__ const int *lhs_words(const adc_ctx &c) { return (const int *)(c.flags + 1); }

// A pending drift made to apply now (before COEF is copied to the host).
__global__ void k_lhs_drift(adc_ctx c) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (lhs_words(c)[1] && i < c.np) row_drift(c, i);
}

__global__ void k_lhs_drift_done(adc_ctx c) {
  griddep_wait();
  int *w = (int *)(c.flags + 1);
  if (w[1]) w[3] = 1;   // the drift changed every row's off-diagonals
  w[1] = 0;
}

// Element pass: matrix entries of the elements that change, or the pending
// drift (kPart 1), the load-vector terms (kPart 2), or both (kPart 3).
// Blocks of the load-vector terms: 64 threads, so that one block's gathers run
// under another's arithmetic (600k nodes: 82 us, 88 with blocks of 256, 83
// with 128), and a small mesh spreads over more SMs.  80 registers a thread
// for half as many warps again was slower, 103 us.
constexpr int kElemThreads = 64;
constexpr int elem_threads(int part) { return part == 1 ? kThreads : kElemThreads; }

template <class R, int kPart>
__global__ void __launch_bounds__(elem_threads(kPart), kPart == 1 ? 4 : kThreads / kElemThreads * (sizeof(R) == 4 ? 3 : 2))
    k_gwce_elem(adc_ctx c) {
  griddep_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (kPart & 1) {
    if (c.flags->ncchange > 0) {
      if (t < c.ne) elem_lhs<R>(c, t);
    } else if (lhs_words(c)[1] && t < c.np) {
      row_drift(c, t);
    }
  }
  if (kPart & 2) {
    __shared__ R sh[kElemThreads / 32][32 * 3];
    const int e0 = t & ~31;
    if (e0 < c.ne) warp_rhs<R>(c, e0, sh[threadIdx.x >> 5]);
  }
}

constexpr int kSMs = 148;

// One kernel for both parts while its blocks run at once (512 threads of 128
// registers on an SM).  Beyond that a second launch costs less than the first
// part's memory passes at the second's occupancy: at 600k nodes 156 us
// together, 21 + 82 us apart; on a small mesh a launch is some 2 us.
template <class R>
static void launch_elem(adc_ctx *c) {
  const int nboth = std::max(c->ne, c->np);
  const int nb = nblk(nboth, kElemThreads);
  kmark(c, KS_LHS_ELEM, 0);
  if (nb <= 2 * (kThreads / kElemThreads) * kSMs) {
    kmark(c, KS_LHS_ELEM, 1);
    kmark(c, KS_RHS_ELEM, 0);
    launch_k(k_gwce_elem<R, 3>, nb, kElemThreads, c->stream, *c);
  } else {
    launch_k(k_gwce_elem<R, 1>, nblk(nboth), kThreads, c->stream, *c);
    kmark(c, KS_LHS_ELEM, 1);
    kmark(c, KS_RHS_ELEM, 0);
    launch_k(k_gwce_elem<R, 2>, nblk(c->ne, kElemThreads), kElemThreads, c->stream, *c);
    c->launches++;
  }
  kmark(c, KS_RHS_ELEM, 1);
}
void launch_gwce_elem(adc_ctx *c) {
  if (f32_assembly(c)) launch_elem<float>(c);   // FP32 element assembly
  else launch_elem<double>(c);
}

// EP = RMS of the diagonal (gwce.F:646-650) from the node blocks' partial
// sums, by 256 threads in the tree of 1,024 (each sums every 1,024th partial
// of four places, then warps, then the 32 warp sums).
__device__ double ep_from_parts(const double *parts, int nparts, int np) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q = 0; q < 4; ++q) {
    double s = 0.0;
    for (int b = threadIdx.x + 256 * q; b < nparts; b += 1024) s += __ldcg(parts + b);
    s = warp_sum(s);
    if (lane == 0) sh[w + 8 * q] = s;
  }
  __syncthreads();
  double s = 0.0;
  if (w == 0) s = warp_sum(sh[lane]);
  return sqrt(s / np);   // valid in thread 0
}

// Node pass.  The last block forms EP and settles the LHS words.
template <class R>
__global__ void __launch_bounds__(kThreads, 4) k_gwce_node(adc_ctx c) {
  griddep_wait();
  const int *words = lhs_words(c);
  const bool rebuild = c.flags->ncchange > 0;
  const int pending = words[1];
  const bool all = words[3] != 0;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double d2 = 0.0;
  if (i < c.np) {
    if (rebuild) d2 = row_lhs<R>(c, i, all);
    node_rhs<R>(c, i);
  }
  __shared__ double sh[32];
  __shared__ int last;
  if (rebuild) {
    d2 = warp_sum(d2);
    if (lane == 0) sh[w] = d2;
    __syncthreads();
    if (w == 0) {
      d2 = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
      d2 = warp_sum(d2);
      if (lane == 0) c.red[blockIdx.x] = d2;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&c.tickets[1], 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double ep = 0.0;
  if (rebuild) ep = ep_from_parts(c.red, gridDim.x, c.np);
  if (threadIdx.x == 0) lhs_settle(c, rebuild, pending, ep);
}

// Boundary rows: matrix rows and columns after a rebuild, then the elevation
// boundary (gwce.F:1638-1651).
__global__ void k_gwce_bc(adc_ctx c, const adc_step_t *steps) {
  griddep_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const double EP = c.flags->ep;
  if (t < c.np + c.n_obc) {
    if (lhs_words(c)[0]) item_bc(c, EP, t);
  } else if (t < c.np + c.n_obc + c.neta) {
    bnd_eta(c, steps[c.flags->cursor], EP, t - c.np - c.n_obc);
  }
}

__global__ void k_obc_rhs(adc_ctx c) {
  griddep_wait();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < c.n_obc_rhs_nodes) bnd_obc(c, r);
}

template __global__ void k_gwce_node<double>(adc_ctx);
template __global__ void k_gwce_node<float>(adc_ctx);

}  // namespace adc
