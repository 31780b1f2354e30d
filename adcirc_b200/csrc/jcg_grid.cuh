// jcg_grid.cuh -- what the two JCG kernels with 256-thread row blocks and a
// scalar block (jcg.cu, jcg_ordered.cu) share: node records, the grid
// barrier that carries the dot products, and the serial scalar steps.
#pragma once

#include "jcg_chgcon.cuh"
#include "jcg_common.cuh"

namespace adc {

// 32-byte node record (dtwd, d, d_prev, -) moved with one 256-bit access.
struct __align__(32) P4 {
  double x, y, z, w;
};

__device__ __forceinline__ P4 ld_p4(const P4 *p) {
  P4 r;
  asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
               : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w)
               : "l"(p));
  return r;
}

__device__ __forceinline__ void st_p4(P4 *p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w)
               : "memory");
}

// ---------------------------------------------------------------- barrier
// Contention-free flag barrier that carries its data, read by every block.
// Each block owns one 128-byte arrival line of four slots, used in turn by
// the barrier generations (slot g & 3); a row block posts its three partial
// sums there, the scalar block (the last block of the grid) posts the
// eigenvalue estimate cme that its chgcon produced for this barrier.  An
// empty word holds kEmpty, a signalling-NaN bit pattern no arithmetic
// produces.  Every block polls all arrival lines until each word of the
// current slot is filled, sums the row blocks' partials in one fixed order
// (the same in every block, so every block holds the same bits) and runs
// the serial ITPACK step (pstop_nrms, parcon) itself on its own copy of the
// ITPACK scalars: one L2 round trip both signals and delivers, and no
// release step follows.  A block empties its own slot (g + 2) & 3 when it
// posts generation g: every reader of generation g - 2 has finished
// reading before any block can post generation g (it first had to see
// everyone's generation g - 1 arrival).  Every word is an aligned 8-byte
// access (single-copy atomic); waits are bounded.
constexpr unsigned long long kEmpty = 0x7FF4DEADBEEF0001ull;

struct alignas(128) ArriveLine {
  unsigned long long slot[4][4];   // (p0, p1, p2, -) of a row block; (cme, 0, 0, -) of the scalar block
};

__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ double bitsd(unsigned long long u) {
  return __longlong_as_double((long long)u);
}

// Release/acquire fence at GPU scope: orders a block's results before the
// barrier words it writes, and the words it polled before what it reads next.
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Polls the first N words of a slot until all are filled; v receives them.  A
// poll is one load of the slot's 32 bytes (each word is single-copy atomic by
// itself): with one load per word, and the timeout flag read beside them, the
// 296 x 296 polls of a barrier took 10,200 cycles of an iteration's 16,700 at
// 100k rows (200 mixed-mode steps 58.5 -> 50.7 ms with this).  Bounded: the
// limit and the flag are looked at once in spin_mask + 1 polls.
template <int N>
__device__ inline bool poll_full(volatile unsigned long long *p, unsigned long long (&v)[N], const JcgArgs &a) {
  const long long t0 = clock64();
  for (unsigned m = 1;; ++m) {
    bool full = true;
    unsigned long long w[4];
    asm volatile("ld.relaxed.gpu.global.v4.b64 {%0,%1,%2,%3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(p)
                 : "memory");
#pragma unroll
    for (int k = 0; k < N; ++k) {
      v[k] = w[k];
      full = full && (v[k] != kEmpty);
    }
    if (full) return true;
    if ((m & a.spin_mask) != 0) continue;
    if (*(volatile int *)&a.flags->timeout) return false;
    if (clock64() - t0 > a.spin) {
      atomicExch(&a.flags->timeout, 1);
      return false;
    }
  }
}

__device__ inline Rec read_rec(const Rec *r) {
  const volatile Rec *v = r;
  Rec o;
  o.c1 = v->c1;
  o.c2 = v->c2;
  o.c3 = v->c3;
  o.c4 = v->c4;
  o.halt = v->halt;
  o.need_unorm = v->need_unorm;
  o.in = v->in;
  o.pad_ = 0;
  return o;
}

// pstop_nrms (itpackv.F:809-890, iflag = 1) for iteration `in`.
__device__ inline int pstop_d(ItpLocal *it, int in, double unrm, double dnrm) {
  double con = it->cme, uold, tr, tl;
  if (in < 1) {
    it->q1 = 0;
    it->udnm = 1.0;
    it->stptst = 1000.0;
  }
  if (!it->q1 && !((in > 5) && (in % 5 != 0))) {
    uold = it->udnm;
    it->udnm = unrm;
    if (it->udnm == 0.0) it->udnm = 1.0;
    if ((in > 5) && (fabs(it->udnm - uold) <= it->udnm * it->zeta)) it->q1 = 1;
  }
  tr = sqrt(it->udnm);
  tl = 1.0;
  if (con != 1.0) {
    tl = sqrt(dnrm);
    tr = tr * (1.0 - con);
  }
  it->stptst = tl / tr;
  if (tl >= tr * it->zeta) return 0;
  return 1;
}

// parcon (itpackv.F:1774-1851) for iteration `in`.
__device__ inline void parcon_d(ItpLocal *it, int in, double dtnrm, double c[4]) {
  double rhoold = it->rho;
  double gamold = it->gamma;
  it->gamma = 1.0 / (1.0 - dtnrm / it->delnnm);
  it->rho = 1.0;
  if (in != 0) it->rho = 1.0 / (1.0 - it->gamma * it->delnnm / (gamold * it->delsnm * rhoold));
  it->delsnm = it->delnnm;
  it->gamold = gamold;
  it->rhoold = rhoold;
  c[0] = it->rho * it->gamma;
  c[1] = it->rho;
  c[2] = 1.0 - it->rho;
  c[3] = it->rho * (1.0 - it->gamma);
}

// ------------------------------------------------------------ reductions
// Block-level fixed-tree sum of up to 3 values; result valid in thread 0.
__device__ inline void block_sum3(double &a, double &b, double &c) {
  __shared__ double sh[3][32];
  a = warp_sum(a);
  b = warp_sum(b);
  c = warp_sum(c);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { sh[0][wid] = a; sh[1][wid] = b; sh[2][wid] = c; }
  __syncthreads();
  if (wid == 0) {
    a = lane < nw ? sh[0][lane] : 0.0;
    b = lane < nw ? sh[1][lane] : 0.0;
    c = lane < nw ? sh[2][lane] : 0.0;
    a = warp_sum(a);
    b = warp_sum(b);
    c = warp_sum(c);
  }
  __syncthreads();
}

// One barrier of generation g for every block.  Row blocks post their
// block sums of (p0, p1, p2), the scalar block posts `cme`; then every block
// gathers the row blocks' posts in block order (thread t takes blocks t,
// t + blockDim, ...; then a fixed tree) and thread 0 runs
// `serial(s0, s1, s2, cme)`.  Returns false on timeout.
template <class F>
__device__ inline bool grid_phase(const JcgArgs &a, bool scalar_block, unsigned g, double p0, double p1,
                           double p2, double cme, F serial) {
  __shared__ int bad;
  __shared__ double s_cme;
  const int sl = g & 3, sl_old = (g + 2) & 3;
  if (!scalar_block) block_sum3(p0, p1, p2);
  if (threadIdx.x == 0) {
    bad = 0;
    volatile unsigned long long *own = ((ArriveLine *)a.arrive + blockIdx.x)->slot[0];
    own[4 * sl_old + 0] = kEmpty;
    own[4 * sl_old + 1] = kEmpty;
    own[4 * sl_old + 2] = kEmpty;
    fence_gpu();   // the block's results (and the emptied slot) before its arrival
    if (scalar_block) {
      own[4 * sl + 0] = dbits(cme);
      own[4 * sl + 1] = 0ull;
      own[4 * sl + 2] = 0ull;
    } else {
      own[4 * sl + 0] = dbits(p0);
      own[4 * sl + 1] = dbits(p1);
      own[4 * sl + 2] = dbits(p2);
    }
  }
  __syncthreads();
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  for (int b = threadIdx.x; b <= a.nrb; b += blockDim.x) {
    volatile unsigned long long *ap = ((ArriveLine *)a.arrive + b)->slot[sl];
    unsigned long long v[3];
    if (!poll_full<3>(ap, v, a)) {
      bad = 1;
      break;
    }
    if (b == a.nrb) {
      s_cme = bitsd(v[0]);
    } else {
      s0 += bitsd(v[0]);
      s1 += bitsd(v[1]);
      s2 += bitsd(v[2]);
    }
  }
  fence_gpu();
  __syncthreads();
  if (bad) return false;
  block_sum3(s0, s1, s2);
  if (threadIdx.x == 0) serial(s0, s1, s2, s_cme);
  __syncthreads();
  return true;
}

// Reducing phase end: `serial(s0, s1, s2, cme)` runs in every block on the
// same sums.
template <class F>
__device__ inline bool phase_reduce(const JcgArgs &a, bool scalar_block, unsigned &g, double p0,
                             double p1, double p2, double cme, F serial) {
  ++g;
  return grid_phase(a, scalar_block, g, p0, p1, p2, cme, serial);
}

// Plain barrier (no partials, no record).
__device__ inline bool phase_sync(const JcgArgs &a, bool scalar_block, unsigned &g) {
  ++g;
  return grid_phase(a, scalar_block, g, 0.0, 0.0, 0.0, 0.0, [](double, double, double, double) {});
}

}  // namespace adc
