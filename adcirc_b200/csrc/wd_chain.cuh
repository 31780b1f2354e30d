// wd_chain.cuh -- the W1 friction chain (wetdry.F:593-618) on one block.
#pragma once

#include "step_bodies.cuh"

namespace adc {

// The ordered event list is resolved by the whole block, kChainFast events
// at a time.
// With the events in element order, the value event e assigns is
//   val(e) = max(cand(e), prior(a_e), prior(b_e)),
// where prior(x) is val of the latest earlier event touching node x, or
// the TK that x had before the pass.  Each event's two predecessors are
// found by a backward search; the values then follow by repeated
// max-propagation along those edges until nothing changes (at most the
// depth of the event DAG, each edge pointing to an earlier event), and the
// last event touching a node writes it.  Max is exact, so this equals the
// sequential result bit for bit.

struct ChainSmem {
  int a[kChainFast], b[kChainFast];   // the event's two nodes
  double v[kChainFast];               // candidate, then the value it assigns
  short pa[kChainFast], pb[kChainFast];
  unsigned char lasta[kChainFast], lastb[kChainFast];
  int ord[kChainFast];                // the event's element (its order)
  unsigned long long key[2 * kChainFast];   // (node, order, slot, side) sort keys
};

// k_wd_chain's working set (file scope, so its accesses compile to
// shared-memory instructions).
__shared__ ChainSmem g_chain;

// One chunk of the ordered list.  With `loaded` the chunk's nodes and
// candidates are already in shared memory, else they come from la/lb/lc.
__device__ inline void chain_block(const adc_ctx &c, const int *la, const int *lb, const double *lc,
                            int total, bool loaded) {
  int *s_a = g_chain.a, *s_b = g_chain.b;
  double *s_v = g_chain.v;
  short *s_pa = g_chain.pa, *s_pb = g_chain.pb;
  unsigned char *s_lasta = g_chain.lasta, *s_lastb = g_chain.lastb;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    if (!loaded) {
      s_a[e] = la[e];
      s_b[e] = lb[e];
      s_v[e] = lc[e];   // the event's candidate
      g_chain.ord[e] = e;
    }
    s_lasta[e] = 1;
    s_lastb[e] = 1;
  }
  __syncthreads();
  // predecessors: sort the (node, event, side) pairs; the entry before a
  // pair in sorted order, if it has the same node, is the latest earlier
  // event on that node (bitonic sort in shared memory)
  unsigned long long *key = g_chain.key;
  const int nk = 2 * total;
  int P = 1;
  while (P < nk) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    unsigned long long k = ~0ull;   // padding sorts last
    if (i < nk) {
      const int e = i >> 1, side = i & 1;
      const unsigned long long node = (unsigned)(side ? s_b[e] : s_a[e]);
      k = (node << 33) | ((unsigned long long)(unsigned)g_chain.ord[e] << 12) |
          ((unsigned long long)e << 1) | (unsigned long long)side;
    }
    key[i] = k;
  }
  __syncthreads();
  // thread i holds key i (P <= 2 * kChainFast <= 2 * blockDim.x: two keys
  // per thread at most); partners within a warp trade by shuffle, others
  // through shared memory
  for (int kk = 2; kk <= P; kk <<= 1)
    for (int j = kk >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        for (int i = threadIdx.x; i < P; i += blockDim.x) {
          const int ixj = i ^ j;
          if (ixj > i) {
            const unsigned long long x = key[i], y = key[ixj];
            const bool up = (i & kk) == 0;
            if ((x > y) == up) {
              key[i] = y;
              key[ixj] = x;
            }
          }
        }
        __syncthreads();
      } else {
        // runs of intra-warp stages: every thread updates its own keys
        for (int i0 = threadIdx.x & ~31; i0 < P; i0 += blockDim.x) {
          const int i = i0 + (threadIdx.x & 31);
          unsigned long long x = key[i];
          for (int jj = j; jj > 0; jj >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, jj);
            const bool up = (i & kk) == 0, lower = (i & jj) == 0;
            // the lower partner keeps the min when sorting up, the max otherwise
            const bool keep_min = (lower == up);
            x = keep_min ? (x < y ? x : y) : (x > y ? x : y);
          }
          key[i] = x;
        }
        __syncthreads();
        break;   // the intra-warp stages of this kk are done
      }
    }
  for (int i = threadIdx.x; i < nk; i += blockDim.x) {
    const unsigned long long k = key[i];
    const int e = (int)((k >> 1) & 2047), side = (int)(k & 1);
    int pred = -1;
    if (i > 0 && (key[i - 1] >> 33) == (k >> 33)) pred = (int)((key[i - 1] >> 1) & 2047);
    if (side) s_pb[e] = (short)pred;
    else s_pa[e] = (short)pred;
  }
  __syncthreads();
  // initial values, one thread per event so the global loads overlap
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    double v = s_v[e];
    if (s_pa[e] < 0) {
      const double t = c.tk[s_a[e]];
      if (t > v) v = t;
    }
    if (s_pb[e] < 0) {
      const double t = c.tk[s_b[e]];
      if (t > v) v = t;
    }
    s_v[e] = v;
  }
  __syncthreads();
  // a predecessor found for node x is no longer the last event touching x;
  // each (predecessor, node) pair has one such later event at most
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int pa = s_pa[e], pb = s_pb[e];
    if (pa >= 0) {
      if (s_a[pa] == s_a[e]) s_lasta[pa] = 0;
      else s_lastb[pa] = 0;
    }
    if (pb >= 0) {
      if (s_a[pb] == s_b[e]) s_lasta[pb] = 0;
      else s_lastb[pb] = 0;
    }
  }
  // max-propagation along the predecessor edges (values only grow; a round
  // in which nothing changes is the fixed point); bounded by the list length
  for (int round = 0; round <= total; ++round) {
    int changed = 0;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int pa = s_pa[e], pb = s_pb[e];
      double v = s_v[e];
      double nv = v;
      if (pa >= 0 && s_v[pa] > nv) nv = s_v[pa];
      if (pb >= 0 && s_v[pb] > nv) nv = s_v[pb];
      if (nv != v) {
        s_v[e] = nv;
        changed = 1;
      }
    }
    if (!__syncthreads_or(changed)) break;
  }
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const double v = s_v[e];
    if (s_lasta[e]) {
      const int a = s_a[e];
      c.tk[a] = v;
      c.tkm[3 * a] = v;
      c.tkm[3 * a + 1] = v;
    }
    if (s_lastb[e]) {
      const int b = s_b[e];
      c.tk[b] = v;
      c.tkm[3 * b] = v;
      c.tkm[3 * b + 1] = v;
    }
  }
}

// Sequential-semantics resolution of the W1 TK events by one thread block of
// up to 1,024 threads.
__device__ inline void block_chain(const adc_ctx &c) {
  __shared__ int s_any;
  if (threadIdx.x == 0) s_any = c.flags->n_w1_events;
  __syncthreads();
  if (s_any == 0) return;
  if (s_any <= kChainFast && c.ne < (1 << 21)) {
    // the unordered list W1 wrote: its element tags give the order
    const int total = s_any;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      g_chain.a[e] = c.evu_i[3 * e];
      g_chain.b[e] = c.evu_i[3 * e + 1];
      g_chain.ord[e] = c.evu_i[3 * e + 2];
      g_chain.v[e] = c.evu_c[e];
    }
    __syncthreads();
    chain_block(c, nullptr, nullptr, nullptr, total, true);
    return;
  }
  // long lists: ordered by an exclusive scan of the per-block counts (fixed
  // partition per thread), then resolved in chunks
  const int nb = c.ev_blocks;
  const int T = blockDim.x;
  const int per = (nb + T - 1) / T;
  const int b0 = threadIdx.x * per, b1 = min(nb, b0 + per);
  int mysum = 0;
  for (int b = b0; b < b1; ++b) mysum += c.ev_cnt[b];
  int *sc = (int *)g_chain.key;   // scan scratch, free until the chunks start
  sc[threadIdx.x] = mysum;
  __syncthreads();
  for (int o = 1; o < T; o <<= 1) {
    int v = (threadIdx.x >= (unsigned)o) ? sc[threadIdx.x - o] : 0;
    __syncthreads();
    sc[threadIdx.x] += v;
    __syncthreads();
  }
  const int base = sc[threadIdx.x] - mysum;
  const int total = sc[T - 1];
  // exclusive event offsets of every W1 block (off[nb] = total), then the
  // blocks' events copied into one ordered list by whole warps at a time
  int *off = c.ev_cnt + nb + 1;
  {
    int o = base;
    for (int b = b0; b < b1; ++b) {
      off[b] = o;
      o += c.ev_cnt[b];
    }
    if (threadIdx.x == 0) off[nb] = total;
  }
  __syncthreads();
  int *la = (int *)c.ebuf2;      // ebuf2 holds 3*NE doubles: 2*NE ints, then NE doubles
  int *lb = la + c.ne;
  double *lc = c.ebuf2 + c.ne;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = T >> 5;
  constexpr int kGroup = 8;   // chunks of 32 blocks whose offsets load together
  for (int g0 = warp * 32; g0 < nb; g0 += kGroup * nwarps * 32) {
    int og[kGroup], ng[kGroup];
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int b = g0 + q * nwarps * 32 + lane;
      og[q] = 0;
      ng[q] = 0;
      if (b < nb) {
        og[q] = off[b];
        ng[q] = off[b + 1] - og[q];
      }
    }
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int bw = g0 + q * nwarps * 32;
      const int o0 = og[q], n = ng[q];
      unsigned m = __ballot_sync(0xffffffffu, n > 0);
      while (m) {
        const int j = __ffs(m) - 1;
        m &= m - 1;
        const int jo = __shfl_sync(0xffffffffu, o0, j), jn = __shfl_sync(0xffffffffu, n, j);
        for (int k = lane; k < jn; k += 32) {
          const int src = (bw + j) * kW1Block + k, p = jo + k;
          const int ea = c.ev_a[src], eb = c.ev_b[src];
          const double ec = c.ev_c[src];
          if (p < kChainFast) {   // the first chunk goes straight to shared memory
            g_chain.a[p] = ea;
            g_chain.b[p] = eb;
            g_chain.v[p] = ec;
            g_chain.ord[p] = p;
          } else {
            la[p] = ea;
            lb[p] = eb;
            lc[p] = ec;
          }
        }
      }
    }
  }
  __syncthreads();
  // consecutive chunks of the ordered list; a chunk's first events read the
  // TK the previous chunk left in memory
  for (int s0 = 0; s0 < total; s0 += kChainFast) {
    chain_block(c, la + s0, lb + s0, lc + s0, min(kChainFast, total - s0), s0 == 0);
    __syncthreads();
  }
}

}  // namespace adc
