// jcg_resident.cu -- ITPACK 2D JCG (itpackv.F:63-604) with each row block's
// part of the solve held on its SM.
//
// One 512-thread block per SM: 15 row warps and one scalar warp.  Row warp w
// owns the block's 32-row slices w, w + 15, ..., K at most; dtwd, d(in-1),
// u(in) and u(in-1) of its rows stay in registers for the whole solve, and
// d(in) of the block's rows and of its halo (the foreign rows it reads) in
// shared memory, where the SpMV gathers it.  The scaled matrix (block-local
// 16-bit columns, eight to a 16-byte word, and values) lives in shared memory
// as far as it fits; slices that do not fit are streamed from L2 every
// iteration, one bulk copy per warp in flight, interleaved with resident
// slices.
//
// An iteration is one pass: the 3-term update of the rows (:593-596), the
// SpMV (pjac, :1932-1967), and one exchange that carries the dot products
// and the halo.  A halo row needs only its owner's dtwd: its d(in+1) is
// formed from that and the d(in), d(in-1) the reader already holds, by the
// owner's expression, so both have the same bits.
//
// Exchange, cluster form (kGrid = 0): the whole solve runs in one
// thread-block cluster.  Every block stores its two block sums and the halo
// values that others read straight into their shared memory, with stores
// that report to the receiver's mbarrier; a block goes on when all bytes it
// expects have come.  Measured on B200: about 500 cycles, against 2,700 to
// 3,000 for an all-to-all through L2.
//
// Exchange, grid form (kGrid = 1): each block posts its block sums in a slot
// of its arrival line, and every block polls all lines.  A poll is one
// 32-byte load of a slot, which holds the sums of d.d, d.Ad and u.u; the
// timeout flag, one word for the whole grid, is looked at once in 64 polls.
// (128-bit atomic polls, with a second one for u.u and the flag read beside
// each, made a step 139 us on a 25k-node shelf and 632 on one of 600k; it
// takes 130 and 624.)  An empty word holds kEmpty, a signalling-NaN pattern
// no arithmetic produces.  A line has four slots used in turn; a block empties
// slot (g + 2) & 3 when it posts generation g and checks that this has been
// performed before it posts g + 1.  Readers of g - 2 are done by then (everyone posted g - 1), and
// nobody polls g + 2 before having seen everyone's g + 1.  Each line exists
// twice, for even and odd blocks, which halves the polls per address.  The
// halo word is (dtwd, generation): a reader that finds an older generation
// reads again, so the exchange needs no memory fence.  Generations go on
// from solve to solve.  Every wait is bounded; on expiry the kernel records
// a timeout and all blocks return.
//
// The adaptive eigenvalue estimate (chgcon, :893-1027) feeds only the
// stopping test.  The scalar warp of every block forms bounds of it from the
// recorded parcon coefficients (CmeBounds) and may fall behind the row warps:
// the estimate never decreases, so while the iterate's change is too large to
// stop by an earlier lower bound, it is too large by the exact estimate.  Only
// an iteration for which that does not decide waits for its own bounds, and
// only where the test falls between them does the scalar warp run chgcon
// itself, from the first iteration on.  Run in every iteration, its search is
// the longest chain of a solve on small meshes (6,500 cycles an iteration
// beside the rows' 3,300 on a 4,961-node channel: 110 us a step for 75).  The
// value that a caller sees is formed by jcg_estimate when it is asked for.
//
// u(m) is needed for its norm in the first iterations and then in every
// fifth; in the others it is formed while the exchange is under way.
#include "jcg_common.cuh"
#include "jcg_scalar.cuh"
#include "tma.cuh"

#include <cfloat>
#include <cstring>
#include <vector>
#include <algorithm>

namespace adc {

// 15 row warps and one scalar warp: with a 17th warp the register file
// (16,384 a quarter SM) would leave 96 registers a thread instead of 128.
constexpr int kRowWarps = 15;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kResThreads = kRowThreads + 32;   // the scalar warp
constexpr int kPart = 16;                       // stride of a block's per-warp sums
constexpr int kMaxCluster = 16;
constexpr unsigned long long kEmpty = 0x7FF4DEADBEEF0001ull;
constexpr unsigned long long kNever = 0x7FF4DEADBEEF0003ull;   // in no line, ever

__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ double bitsd(unsigned long long u) {
  return __longlong_as_double((long long)u);
}

struct W2 {
  unsigned long long x, y;
};

__device__ __forceinline__ W2 ld_w2(const void *p) {
  W2 r;
  asm volatile(
      "{\n .reg .b128 r;\n ld.relaxed.gpu.global.b128 r, [%2];\n mov.b128 {%0, %1}, r;\n}\n"
      : "=l"(r.x), "=l"(r.y)
      : "l"(p)
      : "memory");
  return r;
}

__device__ __forceinline__ void st_w2(void *p, unsigned long long x, unsigned long long y) {
  asm volatile(
      "{\n .reg .b128 r;\n mov.b128 r, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], r;\n}\n" ::"l"(p),
      "l"(x), "l"(y)
      : "memory");
}

__device__ __forceinline__ W2 exch_w2(void *p, unsigned long long x, unsigned long long y) {
  W2 r;
  asm volatile(
      "{\n .reg .b128 r, s;\n mov.b128 r, {%3, %4};\n"
      " atom.relaxed.gpu.global.exch.b128 s, [%2], r;\n mov.b128 {%0, %1}, s;\n}\n"
      : "=l"(r.x), "=l"(r.y)
      : "l"(p), "l"(x), "l"(y)
      : "memory");
  return r;
}

// One poll of a slot: its first three words, each single-copy atomic.
__device__ __forceinline__ void poll_slot(const void *p, unsigned long long &x, unsigned long long &y,
                                          unsigned long long &z) {
  [[maybe_unused]] unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(x), "=l"(y), "=l"(z), "=l"(w)
               : "l"(p)
               : "memory");
}

__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// The row warps alone (the scalar warp runs on).
__device__ __forceinline__ void row_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(kRowThreads) : "memory");
}

// The polling warps among themselves.
__device__ __forceinline__ void poll_barrier(int threads) {
  asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory");
}
// The row warps; true in all of them if `x` is nonzero in any thread.
__device__ __forceinline__ bool row_barrier_or(int x) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n barrier.cta.red.or.pred q, 3, %2, p;\n"
      " selp.s32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(x), "n"(kRowThreads)
      : "memory");
  return r != 0;
}
// Stores into another block's shared memory that report their bytes to an
// mbarrier there, and the wait for all bytes of a phase.
__device__ __forceinline__ void st_async(uint32_t a, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async2(uint32_t a, double v, double w, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
      "l"(__double_as_longlong(v)), "l"(__double_as_longlong(w)), "r"(bar)
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Butterfly sum: every lane ends with the same bits.
__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The ITPACK scalars of one solve, in shared memory: parcon's stepped by
// warp 0, pstop's by warp 1, read by the scalar warp.
struct Scal {
  double gamma, rho, gamold, rhoold, delnnm, delsnm, udnm, squd, sqd, tl, tr, con;
  int q1, exact;
};

// What the other warps need of an iteration's serial step.
struct StepRec {
  double c1, c2, c3, c4;
  int halt, need_u;
};

// Groups of eight slots a slice of width w is stored in.
__host__ __device__ __forceinline__ int slot_groups(int w) { return w > 8 ? (w + 7) >> 3 : 1; }

// The SpMV, -sum_q value_q d[col_q] in slot order (pjac's j order).  A
// slice's slots are stored in groups of eight: a 16-byte word of column byte
// offsets per lane, then eight values per lane.  Slots past a row's end point
// at a cell that holds 0, so that no load or product carries a condition.
__device__ __forceinline__ double gather(const unsigned char *x, unsigned off) {
  return *(const double *)(x + off);
}

// Slots H .. H + 3 of the group whose columns are c.
template <int H>
__device__ __forceinline__ void load4(double (&v)[4], double (&xx)[4], const uint4 &c, const double *lv,
                                      const unsigned char *x) {
  const unsigned lo = H == 0 ? c.x : c.z, hi = H == 0 ? c.y : c.w;
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = lv[(H + q) * kSlice];
  xx[0] = gather(x, lo & 0xffffu);
  xx[1] = gather(x, lo >> 16);
  xx[2] = gather(x, hi & 0xffffu);
  xx[3] = gather(x, hi >> 16);
}

__device__ __forceinline__ void sub4(double &acc, const double (&v)[4], const double (&xx)[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) acc = acc - v[q] * xx[q];
}

// Two slices at p0 and p1 (shared memory) side by side: their two chains of
// sums overlap.
__device__ __forceinline__ void pair_spmv(double &acc0, double &acc1, const unsigned char *p0, int ng0,
                                          const unsigned char *p1, int ng1, const unsigned char *x) {
  const int lane = threadIdx.x & 31;
  const uint4 c0 = ((const uint4 *)p0)[lane], c1 = ((const uint4 *)p1)[lane];
  const double *v0 = (const double *)(p0 + ng0 * 512) + lane, *v1 = (const double *)(p1 + ng1 * 512) + lane;
  {
    double a[4], b[4], xa[4], xb[4];
    load4<0>(a, xa, c0, v0, x);
    load4<0>(b, xb, c1, v1, x);
    sub4(acc0, a, xa);
    sub4(acc1, b, xb);
    load4<4>(a, xa, c0, v0, x);
    load4<4>(b, xb, c1, v1, x);
    sub4(acc0, a, xa);
    sub4(acc1, b, xb);
  }
  // rows of more than eight neighbours
#pragma unroll 1
  for (int g = 1; g < max(ng0, ng1); ++g) {
    double a[4], xa[4];
    if (g < ng0) {
      const uint4 c = ((const uint4 *)p0)[g * 32 + lane];
      load4<0>(a, xa, c, v0 + g * 8 * kSlice, x);
      sub4(acc0, a, xa);
      load4<4>(a, xa, c, v0 + g * 8 * kSlice, x);
      sub4(acc0, a, xa);
    }
    if (g < ng1) {
      const uint4 c = ((const uint4 *)p1)[g * 32 + lane];
      load4<0>(a, xa, c, v1 + g * 8 * kSlice, x);
      sub4(acc1, a, xa);
      load4<4>(a, xa, c, v1 + g * 8 * kSlice, x);
      sub4(acc1, a, xa);
    }
  }
}

// A slice wider than the staging buffer, read in place from global memory
// (a few slices of a mesh).
__device__ __forceinline__ double spmv_global(const uint4 *cv, const double *lv, int len,
                                              const unsigned char *x) {
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
#pragma unroll 1
  for (int q = 0; q < len; ++q) {
    const unsigned short *c = (const unsigned short *)(cv + (q >> 3) * 32 + lane);
    acc = acc - lv[q * kSlice + lane] * gather(x, c[q & 7]);
  }
  return acc;
}

// chgcon as far as a scalar warp has run it, and on to iteration `to`; apart,
// so that its registers and code do not lie in every solve's way.
struct Chgcon {
  double cme, cmold;
  int in, adapt, ier;
};
static __device__ __forceinline__ void chgcon_to(Chgcon *c, int to, const double2 *hist, double2 *tri, double zeta,
                                              double tol, int itmax) {
  double cme = c->cme, cmold = c->cmold;
  int in = c->in, adapt = c->adapt, ier = c->ier;
  while (in < to) {
    ++in;
    if (!adapt) continue;
    const double2 h = hist[max(in - 1, 0)], o = hist[max(in - 2, 0)];
    chgcon_warp<false>(h.x, h.y, o.x, o.y, zeta, tol, itmax, tri, in, cme, cmold, adapt, ier);
  }
  c->cme = cme;
  c->cmold = cmold;
  c->in = in;
  c->adapt = adapt;
  c->ier = ier;
}

template <int K, int kGrid>
__global__ void __launch_bounds__(kResThreads, 1) jcg_resident_kernel(JcgArgs a) {
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool row_warp = warp < kRowWarps;
  const int nrb = a.nrb, b = blockIdx.x, n = a.n;
  const int s0 = (int)((long long)a.nslices * b / nrb);
  const int nsl = (int)((long long)a.nslices * (b + 1) / nrb) - s0;
  const int r0 = s0 * kSlice;
  const int RB = a.rows_max;
  const unsigned zcell = 8u * (unsigned)(RB + a.halo_max);
  extern __shared__ __align__(128) unsigned char sm[];
  double *S_d = (double *)sm;                       // d of the rows, of the halo, and a zero
  const unsigned char *const xd = sm;               // S_d by byte offsets
  double *S_hp = (double *)(sm + a.o_hp);           // halo: d(in-1); cluster form: then two
  double *S_rx = S_hp + a.halo_max;                 // buffers of received values
  int *S_hid = (int *)(sm + a.o_hid);               // halo: global row, or (rank << 16) | local row
  double2 *tri = (double2 *)(sm + a.o_tri);         // the scalar warp's tridiagonal
  double2 *hist = tri + a.itmax + 2;                // (gamma, rho) of every iteration
  int4 *S_meta = (int4 *)(sm + a.o_meta);
  double *S_part = (double *)(sm + a.o_part);
  uint64_t *S_bar = (uint64_t *)(sm + a.o_bar);
  // One area in three roles: w of the prologue; then the staging buffers, or
  // (cluster form) the rows' exported values of two exchanges.
  double *S_w = (double *)(sm + a.o_area);
  double *S_x = (double *)(sm + a.o_area);
  unsigned char *stage = sm + a.o_area + (size_t)(2 * warp) * a.stage_bytes;   // two buffers
  __shared__ Scal sc;
  __shared__ StepRec s_rec;
  __shared__ volatile double s_low, s_up;  // the scalar warp's bounds of the estimate ...
  __shared__ volatile int s_cme_m;         // ... and their iteration (-1: none yet)
  __shared__ volatile double s_con;        // the exact estimate, of the iteration
  __shared__ volatile int s_exact_m;       // s_exact_m, where it is known or
  __shared__ volatile int s_want;          // was asked for
  __shared__ volatile int s_hist;          // iterations recorded in hist
  __shared__ volatile int s_done;          // 1: the solve has ended, 2: a wait expired
  __shared__ int s_m;
  // Cluster form: the bytes of an exchange, alternating: a block whose own
  // exchange is complete may send the next one's before ours is.
  __shared__ uint64_t s_xbar[2];

  const int h0 = a.halo_ptr[b], nhalo = a.halo_ptr[b + 1] - h0;
  // cluster form: the values this block sends (row, receiver and place)
  const int q0 = kGrid ? 0 : a.push_ptr[b], npush = kGrid ? 0 : a.push_ptr[b + 1] - q0;
  int2 *S_push = (int2 *)(sm + a.o_push);
  // echall (itpackv.F:1212-1255) and the zeta floor of jcg (:223-232)
  double zeta = a.run_init ? a.itp->rparm1 : a.itp->zeta;
  if (a.run_init && zeta < 512.0 * DBL_EPSILON) zeta = 512.0 * DBL_EPSILON;
  const int q1_in = a.itp->q1;
  unsigned ag = kGrid ? a.bar->count : 0u, tag = kGrid ? a.bar->gen : 0u;

  // From five slices per warp on, u lives in global memory (u1 for even
  // iterates, u for odd ones): four vectors of nine rows would not fit the
  // registers.
  constexpr bool kUGlobal = K > 4;
  constexpr int KU = kUGlobal ? 1 : K;
  double t[K], dp[K], u[KU], up[KU], pu0 = 0.0;
  // Up to two slices per warp: a row's first group of columns and values
  // stays in registers too.
  constexpr bool kRegs = K <= 2;
  constexpr int KM = kRegs ? K : 1;
  double mv[KM][8];
  uint4 mc[KM];
  unsigned le[(K + 3) / 4];
#pragma unroll
  for (int k = 0; k < (K + 3) / 4; ++k) le[k] = 0u;
#define LE(k) ((le[(k) >> 2] >> (((k) & 3) * 8)) & 0xffu)

  // ---- prologue: scal part 1 (itpackv.F:2281-2421) -- u' = u sqrt(d),
  // w = 1/sqrt(d), rhs' = rhs w.  t holds rhs' until the first SpMV.
  if (row_warp) {
    double dg[K], uu[K], rh[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, i = r0 + ls * kSlice + lane;
      if (ls < nsl && i < n) {
        dg[k] = a.diag[i];
        uu[k] = a.u[i];
        rh[k] = a.rhs[i];
        le[k >> 2] |= (unsigned)a.rle[i] << ((k & 3) * 8);
      }
    }
    for (int s = tid; s < nsl; s += kRowThreads) S_meta[s] = a.meta[s0 + s];
    for (int h = tid; h < nhalo; h += kRowThreads) S_hid[h] = a.halo_ids[h0 + h];
    for (int q = tid; q < npush; q += kRowThreads) S_push[q] = a.push[q0 + q];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, idx = ls * kSlice + lane, i = r0 + idx;
      t[k] = 0.0;
      if constexpr (!kUGlobal) u[k] = 0.0;
      if (ls < nsl && i < n) {
        const double work = sqrt(dg[k]);
        const double us = uu[k] * work;
        const double wv = 1.0 / work;
        const double rs = rh[k] * wv;
        a.w[i] = wv;
        if (a.do_peror) ((double *)a.p0)[2 * (size_t)a.nslices * kSlice + i] = rs;
        a.rhs[i] = rs * (1.0 / wv);   // as unscal leaves it (:2447-2477)
        S_d[idx] = us;
        S_w[idx] = wv;
        if constexpr (kUGlobal) a.u1[i] = us;
        else u[k] = us;
        pu0 += us * us;
        t[k] = rs;
      }
    }
    for (int h = tid; h < nhalo; h += kRowThreads) {
      const int id = S_hid[h];   // written by this thread
      const int j = kGrid ? id
                          : (int)((long long)a.nslices * (id >> 16) / nrb) * kSlice + (id & 0xffff);
      // the owner's expressions on the raw guess and diagonal, which no
      // block overwrites before its epilogue, after the first exchange
      const double work = sqrt(a.diag[j]);
      S_d[RB + h] = a.u[j] * work;
      S_w[RB + h] = 1.0 / work;
    }
  }
  if (tid < (kGrid ? 6 : 9) * kPart) S_part[tid] = 0.0;   // sums of absent warps and blocks stay 0
  if (tid == 0) S_d[zcell >> 3] = 0.0;
  if (!kGrid && tid < 2) mbar_init(&s_xbar[tid], 1);
  if (tid < 2 * kRowWarps) mbar_init(&S_bar[tid], 1);
  mbar_fence_init();
  __syncthreads();

  // ---- scal part 2: scaled off-diagonals (kept in shared memory where the
  // slice is resident), the unscal drift of COEF, d0 = pjac(u') + rhs' - u'.
  // The first group of a warp's next slice is requested before the current
  // slice is worked on.
  if (row_warp) {
    uint4 cn = make_uint4(0u, 0u, 0u, 0u);
    double vn[8];
    auto request = [&](int ls, int g, uint4 &c, double (&v)[8]) {
      if (ls < nsl) {
        const int4 mt = S_meta[ls];
        c = a.rcol[((size_t)mt.z + g) * 32 + lane];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (8 * g + q < mt.y) v[q] = a.offd[mt.x + (8 * g + q) * kSlice + lane];
      }
    };
    request(warp, 0, cn, vn);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, idx = ls * kSlice + lane, i = r0 + idx;
      uint4 c = cn;
      double vo[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) vo[q] = vn[q];
      if (k + 1 < K) request(ls + kRowWarps, 0, cn, vn);
      if constexpr (kRegs) {
        mc[k] = make_uint4(zcell | (zcell << 16), zcell | (zcell << 16), zcell | (zcell << 16),
                           zcell | (zcell << 16));
#pragma unroll
        for (int q = 0; q < 8; ++q) mv[k][q] = 0.0;
      }
      if (ls < nsl) {
        const int4 mt = S_meta[ls];
        const int w = mt.y, len = (int)(LE(k) & 127u), ng = slot_groups(w);
        const bool res = mt.w >= 0;
        const bool glob = !res || a.do_peror;
        unsigned char *rs = sm + a.o_res + (res ? mt.w : 0);
        const double wi = S_w[i < n ? idx : 0];
        double acc = t[k];
        const double ui = i < n ? S_d[idx] : 0.0;
        for (int g = 0; g < ng; ++g) {
          if (g > 0) request(ls, g, c, vo);   // rows of more than eight neighbours
          if constexpr (kRegs)
            if (g == 0) mc[k] = c;
          if (res) ((uint4 *)rs)[g * 32 + lane] = c;
          const unsigned cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int slot = 8 * g + q;
            const unsigned off = q & 1 ? cc[q >> 1] >> 16 : cc[q >> 1] & 0xffffu;
            double sv = 0.0;
            if (slot < len) {
              const double wj = gather((const unsigned char *)S_w, off);
              const double s = vo[q] * wi * wj;
              if (!a.defer_drift) a.offd[mt.x + slot * kSlice + lane] = s * (1.0 / wi) * (1.0 / wj);
              acc = acc - s * gather(xd, off);
              sv = s;
            }
            if constexpr (kRegs)
              if (g == 0) mv[k][q] = sv;
            if (res) ((double *)(rs + ng * 512))[slot * kSlice + lane] = sv;
            if (glob && slot < w) a.soff[mt.x + slot * kSlice + lane] = sv;
          }
        }
        t[k] = acc - ui;   // d0
      }
    }
    fence_proxy_async_all();   // streamed slices are read by bulk copies from here on
  }
  __syncthreads();   // everyone is done with u' and w

  // The warp's streamed slices: bit k set where slice k is streamed.  The
  // q-th of them goes through buffer q & 1, and two copies are in flight,
  // across the exchange too.  With kRegs none is: what is not resident has no
  // slots beyond the registers'.
  unsigned smask = 0u;
  uint32_t bar_par = 0u;
  int bad = 0;   // an expired wait of this thread
  if (row_warp && !kRegs) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps;
      if (ls < nsl && S_meta[ls].w == -1) smask |= 1u << k;
    }
  }
  unsigned s_rem = smask;            // the slices still to copy in this round
  unsigned s_cnt = 0u, l_cnt = 0u;   // copies issued, copies landed
  auto issue = [&]() {   // copies the next streamed slice into its buffer
    const int k = __ffs(s_rem) - 1;
    if (lane == 0) {
      const int4 mt = S_meta[warp + k * kRowWarps];
      const uint32_t cb = (uint32_t)slot_groups(mt.y) * 512u;
      const uint32_t vb = (uint32_t)mt.y * 32u * (uint32_t)sizeof(double);
      const int st = (int)(s_cnt & 1u);
      uint64_t *const bar = &S_bar[2 * warp + st];
      unsigned char *const dst = stage + st * a.stage_bytes;
      mbar_expect_tx(bar, cb + vb);
      bulk_load(dst, a.rcol + (size_t)mt.z * 32, cb, bar);
      if (vb) bulk_load(dst + cb, a.soff + mt.x, vb, bar);
    }
    ++s_cnt;
    s_rem &= s_rem - 1u;
    if (s_rem == 0u) s_rem = smask;
  };
  // waits for the oldest copy in flight: its buffer (kDrainCycles more when
  // the wait has expired, so that no copy outlives the block)
  auto land = [&]() -> int {
    const int st = (int)(l_cnt & 1u);
    const long long tw = clock64();
    while (!mbar_try_wait(&S_bar[2 * warp + st], (bar_par >> st) & 1u)) {
      if (clock64() - tw > a.spin) {
        if (lane == 0) atomicExch(&a.flags->timeout, 1);
        bad = 1;
        if (clock64() - tw - kDrainCycles > a.spin) break;
      }
    }
    bar_par ^= 1u << st;
    ++l_cnt;
    return st;
  };
  if (smask) {
    // slots past a slice's end multiply what the buffer holds by zero: it
    // must hold numbers (see staged_values)
    for (int q = lane; q < 2 * a.stage_bytes / 16; q += 32) ((uint4 *)stage)[q] = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_all();
    __syncwarp();
    issue();
    issue();
  }

  // d0 of the rows and of the halo
  void *const X[2] = {(void *)a.p0, (void *)a.p1};   // grid form: one 16-byte word per row
  ++tag;
  if (row_warp) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, idx = ls * kSlice + lane, i = r0 + idx;
      if (ls < nsl && i >= n) S_d[idx] = 0.0;   // rows past the end add nothing to any norm
      if (ls < nsl && i < n) {
        S_d[idx] = t[k];
        if (!kGrid) S_x[RB + idx] = t[k];   // dtwd goes to S_x[idx]
        else if (LE(k) & 128u) st_w2((char *)X[tag & 1] + 16 * (size_t)i, dbits(t[k]), tag);
      }
    }
  }
  // Halo words of the exchange `g`: the value, polled until it has arrived.
  auto halo_wait = [&](const char *p, W2 q, unsigned g) -> double {
    if (q.y != g) {
      const long long tw = clock64();
      unsigned polls = 0;
      do {
        q = ld_w2(p);
        if (q.y != g && (++polls & a.spin_mask) == 0 &&
            (clock64() - tw > a.spin || *(volatile int *)&a.flags->timeout)) {
          atomicExch(&a.flags->timeout, 1);
          bad = 1;
          break;
        }
      } while (q.y != g);
    }
    return bitsd(q.x);
  };
  __syncwarp();
  if (!kGrid) cluster_barrier();
  if (row_warp) {
    for (int h = tid; h < nhalo; h += kRowThreads) {
      double v;
      if (kGrid) {
        const char *p = (const char *)X[tag & 1] + 16 * (size_t)S_hid[h];
        v = halo_wait(p, ld_w2(p), tag);
      } else {
        v = ld_cluster(cluster_addr(S_x + RB + (S_hid[h] & 0xffff), S_hid[h] >> 16));
      }
      S_d[RB + h] = v;
      S_hp[h] = 0.0;   // d(-1)
    }
  }

  if (tid == 0) {
    memset(&sc, 0, sizeof(sc));
    sc.q1 = q1_in;
    s_cme_m = s_exact_m = s_want = -1;
    s_hist = 0;
    s_done = 0;
  }
  __syncthreads();

  int m = 0;
  bool ended = false;             // the solve has ended, without an expired wait in this block
  unsigned e = 0;                 // exchanges so far: parity of the double buffers
  if (row_warp) {
#pragma unroll
    for (int k = 0; k < K; ++k) dp[k] = 0.0;
#pragma unroll
    for (int k = 0; k < KU; ++k) up[k] = 0.0;
    double c1 = 0.0, c2 = 0.0, c3 = 0.0, c4 = 0.0;
    int need_u = !q1_in, halt = 0;
    W2 emptied = {0ull, 0ull};      // grid form: old word of the slot this lane emptied last
    W2 hq = {0ull, 0ull};           // the thread's first halo word, requested early
    for (;; ++m) {
      double pd = 0.0, pt = 0.0, pu = m == 0 ? pu0 : 0.0;
      // u(m) = c1 d(m-1) + c2 u(m-1) + c3 u(m-2) (itpackv.F:593-594)
      auto update_u = [&]() {
        if constexpr (kUGlobal) {
          double *const cur = m & 1 ? a.u1 : a.u, *const nxt = m & 1 ? a.u : a.u1;
          double uc[K], uo[K];
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int ls = warp + k * kRowWarps, i = r0 + ls * kSlice + lane;
            uc[k] = uo[k] = 0.0;
            if (ls < nsl && i < n) {
              uc[k] = cur[i];
              if (m > 1) uo[k] = nxt[i];
            }
          }
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int ls = warp + k * kRowWarps, i = r0 + ls * kSlice + lane;
            if (ls < nsl && i < n) {
              const double un = c1 * dp[k] + c2 * uc[k] + c3 * uo[k];
              nxt[i] = un;
              pu += un * un;
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const double un = c1 * dp[k] + c2 * u[k] + c3 * up[k];
            up[k] = u[k];
            u[k] = un;
            pu += un * un;
          }
        }
      };
      if (m > 0) {
        // d(m) from the previous iterates (itpackv.F:595-596)
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int ls = warp + k * kRowWarps, idx = ls * kSlice + lane;
          if (ls < nsl) {
            const double d = S_d[idx];
            S_d[idx] = c1 * t[k] + c4 * d + c3 * dp[k];
            dp[k] = d;
          }
        }
        if (need_u) update_u();
        for (int h = tid; h < nhalo; h += kRowThreads) {
          double v;
          if (kGrid) {
            const char *p = (const char *)X[tag & 1] + 16 * (size_t)S_hid[h];
            v = halo_wait(p, h == tid ? hq : ld_w2(p), tag);
          } else {
            v = S_rx[(e & 1) * a.halo_max + h];
          }
          const double d = S_d[RB + h], o = S_hp[h];
          S_hp[h] = d;
          S_d[RB + h] = c1 * v + c4 * d + c3 * o;
        }
      }
      row_barrier();
      // dtwd(m) = -A' d(m) and the dot products; rows another block reads go out
      ++e;
      ++tag;
      if constexpr (kRegs) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const unsigned cc[4] = {mc[k].x, mc[k].y, mc[k].z, mc[k].w};
          double xx[8], acc = 0.0;
#pragma unroll
          for (int q = 0; q < 8; ++q) xx[q] = gather(xd, q & 1 ? cc[q >> 1] >> 16 : cc[q >> 1] & 0xffffu);
#pragma unroll
          for (int q = 0; q < 8; ++q) acc = acc - mv[k][q] * xx[q];
          const int ls = warp + k * kRowWarps;
          if (ls < nsl && S_meta[ls].y > 8) {
            const int4 mt = S_meta[ls];
            const int ng = slot_groups(mt.y);
            const unsigned char *p = sm + a.o_res + mt.w;
#pragma unroll 1
            for (int g = 1; g < ng; ++g) {
              double av[4], xa[4];
              const uint4 c = ((const uint4 *)p)[g * 32 + lane];
              const double *lv = (const double *)(p + ng * 512) + g * 8 * kSlice + lane;
              load4<0>(av, xa, c, lv, xd);
              sub4(acc, av, xa);
              load4<4>(av, xa, c, lv, xd);
              sub4(acc, av, xa);
            }
          }
          t[k] = acc;
        }
      } else {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
          const int l0 = warp + k * kRowWarps, l1 = k + 1 < K ? l0 + kRowWarps : nsl;
          if (l0 < nsl) {
            const int4 m0 = S_meta[l0], m1 = S_meta[l1 < nsl ? l1 : l0];
            const bool has1 = l1 < nsl;
            // shared-memory places; a missing or unstaged slice repeats the other
            const bool in0 = m0.w != -2, in1 = has1 && m1.w != -2;
            double a0 = 0.0, a1 = 0.0;
            if (in0 || in1) {
              const unsigned char *p0 = stage, *p1 = stage;
              if (in0) p0 = m0.w >= 0 ? sm + a.o_res + m0.w : stage + land() * a.stage_bytes;
              if (in1) p1 = m1.w >= 0 ? sm + a.o_res + m1.w : stage + land() * a.stage_bytes;
              const int g0 = slot_groups((in0 ? m0 : m1).y), g1 = slot_groups((in1 ? m1 : m0).y);
              pair_spmv(a0, a1, in0 ? p0 : p1, g0, in1 ? p1 : p0, g1, xd);
            }
            if (m0.w == -1 || (has1 && m1.w == -1)) {
              __syncwarp();
              if (m0.w == -1) issue();
              if (has1 && m1.w == -1) issue();
            }
            if (m0.w == -2)
              a0 = spmv_global(a.rcol + (size_t)m0.z * 32, a.soff + m0.x, (int)(LE(k) & 127u), xd);
            t[k] = a0;
            if (k + 1 < K) {
              if (has1 && m1.w == -2)
                a1 = spmv_global(a.rcol + (size_t)m1.z * 32, a.soff + m1.x, (int)(LE(k + 1) & 127u), xd);
              t[k + 1] = a1;
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int ls = warp + k * kRowWarps, idx = ls * kSlice + lane, i = r0 + idx;
        if (ls < nsl && i < n) {
          if (!kGrid) S_x[idx] = t[k];
          else if (LE(k) & 128u) st_w2((char *)X[tag & 1] + 16 * (size_t)i, dbits(t[k]), tag);
          const double d = S_d[idx];
          pd += d * d;
          pt += d * t[k];
        }
      }
      // ---- exchange of the dot products: warp sums (pd in lanes 0-15, pt in
      // lanes 16-31, from one butterfly), block sums in warp 0, all blocks
      double *part = S_part, *all = S_part + 3 * kPart;   // [3][16]; grid [3][16], cluster [2][3][16]
      double v = (lane & 16 ? pt : pd) + __shfl_xor_sync(0xffffffffu, lane & 16 ? pd : pt, 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (need_u) pu = warp_sum_all(pu);
      if ((lane & 15) == 0) part[(lane >> 4) * kPart + warp] = v;
      if (need_u && lane == 0) part[2 * kPart + warp] = pu;
      // the last emptying has been performed (its old word is back) before
      // the block posts again
      if (kGrid && warp == kRowWarps - 1 && emptied.x == kNever) bad = 1;
      row_barrier();
      double x = 0.0;   // v: (pd, pt) sums as above; x: pu in lanes 0-15
      if (warp == 0) {
        v = part[lane];
        if (need_u) x = part[2 * kPart + (lane & 15)];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          v += __shfl_xor_sync(0xffffffffu, v, o);
          if (need_u) x += __shfl_xor_sync(0xffffffffu, x, o);
        }
      }
      if (!kGrid) {
        double2 *mine = (double2 *)(all + (e & 1) * 3 * kPart);   // (pd, pt) of every block,
        double *mine_u = (double *)(mine + kPart);                // and pu
        if (warp == 0) {
          const double vd = __shfl_sync(0xffffffffu, v, 0), vt = __shfl_sync(0xffffffffu, v, 16);
          if (lane < nrb) {
            const uint32_t bar = cluster_addr(&s_xbar[e & 1], lane);
            st_async2(cluster_addr(mine + b, lane), vd, vt, bar);
            if (need_u) st_async(cluster_addr(mine_u + b, lane), x, bar);
          }
          if (lane == 0) mbar_expect_tx(&s_xbar[e & 1], (uint32_t)(nrb * (need_u ? 24 : 16) + 8 * nhalo));
        }
        for (int q = tid - 32; q < npush; q += kRowThreads - 32) {   // warp 0 has the sums to send
          if (q < 0) break;
          const int2 w = S_push[q];
          const int r = w.y >> 16;
          st_async(cluster_addr(S_rx + (e & 1) * a.halo_max + (w.y & 0xffff), r), S_x[w.x],
                   cluster_addr(&s_xbar[e & 1], r));
        }
        if (m > 0 && !need_u) update_u();
        const long long tw = clock64();
        while (!mbar_try_wait_cluster(&s_xbar[e & 1], ((e - 1u) >> 1) & 1u)) {
          if (clock64() - tw > a.spin) {
            atomicExch(&a.flags->timeout, 1);
            bad = 1;
            break;
          }
        }
        if (warp < 2) {
          const double2 w = mine[lane & 15];
          v = lane & 16 ? w.y : w.x;
          if (need_u) x = mine_u[lane & 15];
        }
      } else {
        ++ag;
        const int slot = 32 * (int)(ag & 3), slot_old = 32 * (int)((ag + 2) & 3);
        const int nthr = max(64, (min(nrb, kRowThreads) + 31) & ~31);   // polling threads, warps 0 and 1 among them
        // lanes 0-3 of warp 0 post (copy, word); those of the last row warp
        // empty the slot of two generations ago
        char *mine = (char *)a.arrive + ((size_t)(lane & 1) * nrb + b) * 128 + 16 * ((lane >> 1) & 1);
        if (warp == 0) {
          const double vd = __shfl_sync(0xffffffffu, v, 0), vt = __shfl_sync(0xffffffffu, v, 16);
          const double vu = __shfl_sync(0xffffffffu, x, 0);
          if (lane < (need_u ? 4 : 2))
            st_w2(mine + slot, dbits(lane < 2 ? vd : vu), lane < 2 ? dbits(vt) : 0ull);
        } else if (warp == kRowWarps - 1 && lane < 4) {
          emptied = exch_w2(mine + slot_old, kEmpty, kEmpty);
        }
        if (m > 0 && !need_u) update_u();
        if (tid < nthr) {
          // one thread per line and its block's word; sums in block order per thread
          double sd = 0.0, st = 0.0, su = 0.0;
          for (int q = tid; q < nrb; q += kRowThreads) {
            char *line = (char *)a.arrive + ((size_t)(b & 1) * nrb + q) * 128 + slot;
            const long long tw = clock64();
            W2 y, z = {0ull, 0ull};
            for (unsigned polls = 1;; ++polls) {
              poll_slot(line, y.x, y.y, z.x);
              if (y.x != kEmpty && y.y != kEmpty && (!need_u || z.x != kEmpty)) break;
              if ((polls & a.spin_mask) == 0 &&
                  (clock64() - tw > a.spin || *(volatile int *)&a.flags->timeout)) {
                atomicExch(&a.flags->timeout, 1);
                bad = 1;
                break;
              }
            }
            if (!need_u) z.x = 0ull;
            sd += bitsd(y.x);
            st += bitsd(y.y);
            su += bitsd(z.x);
          }
          __syncwarp();
          double s = (lane & 16 ? st : sd) + __shfl_xor_sync(0xffffffffu, lane & 16 ? sd : st, 16);
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (need_u) su = warp_sum_all(su);
          if ((lane & 15) == 0) all[(lane >> 4) * kPart + warp] = s;
          if (need_u && lane == 0) all[2 * kPart + warp] = su;
          poll_barrier(nthr);
        }
        if (warp < 2) {
          const int nw = nthr >> 5;
          v = (lane & 15) < nw ? all[lane] : 0.0;
          if (need_u) x = (lane & 15) < nw ? all[2 * kPart + (lane & 15)] : 0.0;
        }
      }
      // ---- the serial step, in two warps side by side (in every warp its
      // FP64 divisions would take turns on the FP64 pipe)
      if (warp < 2) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          v += __shfl_xor_sync(0xffffffffu, v, o);
          if (need_u) x += __shfl_xor_sync(0xffffffffu, x, o);
        }
        const double sd = __shfl_sync(0xffffffffu, v, 0), st = __shfl_sync(0xffffffffu, v, 16);
        const double su = __shfl_sync(0xffffffffu, x, 0);
        if (warp == 0) {   // parcon (itpackv.F:1774-1851)
          const double g0 = sc.gamma, r0s = sc.rho, P = g0 * sc.delsnm * r0s;
          const double gamma = 1.0 / (1.0 - st / sd);
          const double q = gamma * sd / P;
          const double rho = m != 0 ? 1.0 / (1.0 - q) : 1.0;
          if (lane == 0) {
            s_rec.c1 = rho * gamma;
            s_rec.c2 = rho;
            s_rec.c3 = 1.0 - rho;
            s_rec.c4 = rho * (1.0 - gamma);
            sc.gamold = g0;
            sc.rhoold = r0s;
            sc.gamma = gamma;
            sc.rho = rho;
            sc.delnnm = sc.delsnm = sd;
            s_m = m;
            hist[m] = make_double2(gamma, rho);
          }
        } else {   // pstop_nrms (itpackv.F:809-890, iflag = 1)
          double udnm = sc.udnm, squd = sc.squd;
          int q1 = sc.q1;
          if (m < 1) {
            q1 = 0;
            udnm = 1.0;
            squd = 1.0;
          }
          if (!q1 && !((m > 5) && (m % 5 != 0))) {
            const double uold = udnm;
            udnm = need_u ? su : 1.0;
            if (udnm == 0.0) udnm = 1.0;
            if ((m > 5) && (fabs(udnm - uold) <= udnm * zeta)) q1 = 1;
            squd = sqrt(udnm);
          }
          const double sqd = sqrt(sd);
          // Waits of the scalar warp's; false where the wait expires.
          const auto wait_for = [&](volatile int &at) {
            const long long tw = clock64();
            while (at < m) {
              if (clock64() - tw > a.spin) {
                if (lane == 0) atomicExch(&a.flags->timeout, 1);
                bad = 1;
                return;
              }
            }
            __threadfence_block();
          };
          // an earlier lower bound may decide: con(m) is no smaller, so that
          // tr (1 - con) zeta is no larger (con = 1 does not stop either
          // while squd zeta <= 1)
          const auto goes_on = [&](double low) {
            return m < a.itmax && squd * zeta <= 1.0 && sqd >= squd * (1.0 - low) * zeta;
          };
          int h = 0;
          const int seen = s_cme_m;
          __threadfence_block();
          if (!(m >= 2 && seen >= 1 && goes_on(s_low))) {
            wait_for(s_cme_m);
            bool exact = s_exact_m >= m;
            if (!exact && !goes_on(s_low)) {
              const double up = s_up;
              if (m < a.itmax && up < 1.0 && sqd < squd * (1.0 - up) * zeta) {
                h = 1;
              } else {
                if (lane == 0) s_want = m;
                wait_for(s_exact_m);
                exact = true;
              }
            }
            if (exact) {
              const double con = s_con;
              double tl = 1.0, tr = squd;
              if (con != 1.0) {
                tl = sqd;
                tr = tr * (1.0 - con);
              }
              h = (tl >= tr * zeta) ? 0 : 1;
              if (!h && m >= a.itmax) h = 2;
              if (lane == 0) {
                sc.tl = tl;
                sc.tr = tr;
                sc.con = con;
              }
            }
            if (lane == 0) {
              sc.exact = exact;
              sc.sqd = sqd;
            }
          }
          if (lane == 0) {
            s_rec.halt = h;
            s_rec.need_u = !(q1 || ((m + 1 > 5) && ((m + 1) % 5 != 0)));
            sc.udnm = udnm;
            sc.squd = squd;
            sc.q1 = q1;
          }
        }
      }
      // an expired wait anywhere in the block ends the solve in all its threads
      const bool failed = row_barrier_or(bad);
      halt = s_rec.halt;
      if (failed || halt) {
        if (tid == 0) {
          __threadfence_block();
          s_done = failed ? 2 : 1;
        }
        while (l_cnt != s_cnt) land();   // the copies in flight
        ended = !failed;
        break;
      }
      if (tid == 0) {
        __threadfence_block();
        s_hist = m + 1;   // the scalar warp may form the next estimate
      }
      // every block has posted: the halo words are (nearly) all there
      if (kGrid && tid < nhalo) hq = ld_w2((const char *)X[tag & 1] + 16 * (size_t)S_hid[tid]);
      c1 = s_rec.c1;
      c2 = s_rec.c2;
      c3 = s_rec.c3;
      c4 = s_rec.c4;
      need_u = s_rec.need_u;
    }
  } else {
    const double cmold0 = a.itp->cmold, cme0 = a.itp->cme;
    const int adapt0 = a.run_init ? 1 : a.itp->adapt;
    const double ztol = zbrent_tol(zeta);
    Chgcon ch = {cme0, cmold0, -1, adapt0, 0};
    int ex = -1, adapt = adapt0;   // ch.in and ch.adapt
    CmeBounds bd;
    bd.low = bd.up = 0.0;
    // What the row warps have left in shared memory is read by lane 0 alone:
    // lanes that read it one by one may differ, and all of them go on together.
    int done = 0;   // s_done, where lane 0 last read it
    for (int in = 0;;) {
      int to = -1;   // run chgcon up to here; -2: the end
      if (lane == 0) {
        const long long tw = clock64();
        while (s_hist < in && s_done == 0 && s_want <= ex) {
          if (clock64() - tw > 2 * a.spin) break;   // the row warps have given up before
        }
        done = s_done;
        if (in > 0 && done != 0) to = -2;
        else if (s_want > ex) to = s_want;
        else if (s_hist < in) to = -2;
        __threadfence_block();
      }
      to = __shfl_sync(0xffffffffu, to, 0);
      __syncwarp();   // lane 0's reads before every lane's
      if (to == -2) break;
      // the first two, and all once the estimate stays as it is, cost nothing
      const bool next = to < 0;
      if (next && ex == in - 1 && (in <= 1 || !adapt)) to = in;
      if (ex < to) {
        chgcon_to(&ch, to, hist, tri, zeta, ztol, a.itmax);
        ex = to;
        adapt = ch.adapt;
      }
      if (next) {
        if (ex == in) {
          if (in == 1) bd.start(zeta, s_con, ch.cme);
          else bd.low = bd.up = ch.cme;
        } else {
          const double2 h = hist[in - 1], o = hist[in - 2];
          tri_entries(h.x, h.y, o.x, o.y, tri, in);
          bd.next(zeta, ztol, tri, in);
        }
      }
      if (lane == 0) {
        if (ex == to) {
          s_con = ch.cme;
          __threadfence_block();
          s_exact_m = ex;
        }
        if (next) {
          s_low = bd.low;
          s_up = bd.up;
          __threadfence_block();
          s_cme_m = in;
        }
      }
      __syncwarp();
      if (next) ++in;
    }
    ended = __shfl_sync(0xffffffffu, done, 0) == 1;
    m = s_m;
    if (ended && b == 0 && !sc.exact)
      for (int k = lane; k < m; k += 32) ((double2 *)(a.est + 1))[k] = hist[k];
    if (ended && b == 0 && lane == 0) {
      const Scal s = sc;
      const int halt = s_rec.halt;
      const double stptst = s.exact ? s.tl / s.tr : 0.0;
      double rparm1 = a.itp->rparm1;
      if (halt == 2) rparm1 = stptst;   // itpackv.F:394
      // without the exact estimate, jcg_estimate's inputs
      EstRec *er = a.est;
      er->zeta = zeta; er->cme0 = cme0; er->cmold0 = cmold0; er->sqd = s.sqd; er->squd = s.squd;
      er->m = m; er->itmax = a.itmax; er->adapt0 = adapt0; er->exact = s.exact;
      ++er->serial;
      Itp *g = a.itp;
      g->zeta = zeta; g->cme = s.con; g->gamma = s.gamma; g->rho = s.rho;
      g->gamold = s.gamold; g->rhoold = s.rhoold; g->delnnm = s.delnnm; g->delsnm = s.delsnm;
      g->udnm = s.udnm; g->stptst = stptst; g->cmold = ch.cmold; g->rparm1 = rparm1;
      g->sme = -1.0; g->itmax = a.itmax; g->isym = 0;
      g->adapt = adapt; g->q1 = s.q1; g->chg_ier = ch.ier;
      g->in = m;
      g->halt = halt;
      if (a.defer_drift == 1) *a.drift_pending = 1;
      a.flags->numitr = m;
      a.flags->ier = (halt == 2) ? 13 : 0;
      a.flags->zeta = rparm1;
      a.flags->cme = s.con;
      if (a.d1) a.flags->n_w1_events = 0;
    }
  }

  // ---- epilogue: unscal (itpackv.F:2447-2477), the GWCE eta update
  // (gwce.F:2006-2008) and wet/dry pass D1, which took a launch of 2 us and a
  // second pass over ETA2 and NODECODE by itself
  if (row_warp && ended) {
    double wv[K], e1[K], uf[K], dp[K];
    int nc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, i = r0 + ls * kSlice + lane;
      if (ls < nsl && i < n) {
        wv[k] = a.w[i];
        if constexpr (kUGlobal) uf[k] = (m & 1 ? a.u : a.u1)[i];
        else uf[k] = u[k];
        if (a.eta_update) {
          e1[k] = a.eta1[i];
          nc[k] = a.nodecode[i];
          if (a.d1) dp[k] = a.dp[i];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int ls = warp + k * kRowWarps, i = r0 + ls * kSlice + lane;
      if (ls < nsl && i < n) {
        const double un = uf[k] * wv[k], winv = 1.0 / wv[k];
        if (a.do_peror) a.u1[i] = uf[k];
        a.u[i] = un;
        a.diag[i] = winv * winv;
        if (a.eta_update) {
          double e2 = nc[k] * (un + 0.0) + e1[k];
          if (a.d1 && d1_dries(nc[k], dp[k], a.h0, e2)) {
            a.nnodecode[i] = 0;
            a.nodecode[i] = 0;
            atomicAdd(&a.flags->ncchange, 1);
          }
          a.eta2[i] = e2;
        }
      }
    }
  }
  if (kGrid && ended && b == 0 && tid == 0) {
    a.bar->count = ag;
    a.bar->gen = tag;
  }
  __syncwarp();
  if (!kGrid) {
    // No block leaves while another may read its shared memory or store into
    // it, after an expired wait either: by the barrier every block has issued
    // its last stores (each of its waits is bounded), and they get time to
    // come in, those of the exchange that this block did not complete and
    // those of the next, which a block that did may have begun.
    cluster_barrier();
    if (row_warp && !ended) {
      const long long tw = clock64();
      while (!(mbar_try_wait_cluster(&s_xbar[e & 1], ((e - 1u) >> 1) & 1u) &&
               mbar_try_wait_cluster(&s_xbar[(e + 1u) & 1], (e >> 1) & 1u)) &&
             clock64() - tw < kDrainCycles) {
      }
    }
  }
#undef LE
}

// peror (itpackv.F:607-720): per-block partial sums of the norms behind
// digit1/digit2 from what the solve left (scaled u in u1, scaled rhs beside
// the exchange words, the scaled matrix), then their sum in block order.
// pmult (itpackv.F:1970-2005) forms c = u - sum_j coef(:,j) u(jcoef).
__global__ void jcg_peror_kernel(JcgArgs a, double *part) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double pb = 0.0, pr = 0.0;
  if (i < a.n) {
    const double *rs = (const double *)a.p0 + 2 * (size_t)a.nslices * kSlice;
    const double wv = a.w[i];
    const double wk = rs[i] / wv;
    pb = wk * wk;
    const int s = i / kSlice, base = a.sl_ptr[s] + i % kSlice, len = a.rlen[i];
    double cc = a.u1[i];
    for (int k = 0; k < len; ++k) {
      const int q = base + k * kSlice;
      cc = cc - a.soff[q] * a.u1[a.col[q]];
    }
    const double wk2 = (rs[i] - cc) / wv;
    pr = wk2 * wk2;
  }
  __shared__ double sh[2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  pb = warp_sum_all(pb);
  pr = warp_sum_all(pr);
  if (lane == 0) {
    sh[0][w] = pb;
    sh[1][w] = pr;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      pb += sh[0][k];
      pr += sh[1][k];
    }
    part[2 * blockIdx.x] = pb;
    part[2 * blockIdx.x + 1] = pr;
  }
}

__global__ void jcg_peror_sum(Itp *itp, const double *part, int nparts) {
  griddep_wait();
  double pb = 0.0, pr = 0.0;
  for (int k = threadIdx.x; k < nparts; k += 32) {
    pb += part[2 * k];
    pr += part[2 * k + 1];
  }
  pb = warp_sum_all(pb);
  pr = warp_sum_all(pr);
  if (threadIdx.x == 0) {
    itp->dtnrm = pb;
    itp->unorm = pr;
  }
}

int launch_jcg_peror(const JcgArgs &a, adc_ctx *c) {
  const int nb = nblk(a.n);
  double *part = (double *)a.p1 + 2 * (size_t)a.nslices * kSlice;   // beside the exchange words
  launch_k(jcg_peror_kernel, nb, kThreads, c->stream, a, part);
  launch_k(jcg_peror_sum, 1, 32, c->stream, a.itp, (const double *)part, nb);
  c->launches += 2;
  return ADC_OK;
}

// ------------------------------------------------------------------ host

// The instance for at most `k` slices per warp (nullptr: none).
static const void *res_fn(int k, bool grid) {
  if (!grid)
    return k <= 1   ? (const void *)jcg_resident_kernel<1, 0>
           : k <= 2 ? (const void *)jcg_resident_kernel<2, 0>
                    : nullptr;
  return k <= 1   ? (const void *)jcg_resident_kernel<1, 1>
         : k <= 2 ? (const void *)jcg_resident_kernel<2, 1>
         : k <= 4 ? (const void *)jcg_resident_kernel<4, 1>
         : k <= 6 ? (const void *)jcg_resident_kernel<6, 1>
         : k <= 9 ? (const void *)jcg_resident_kernel<9, 1>
                  : nullptr;
}

static size_t align_up(size_t v, size_t m) { return (v + m - 1) / m * m; }

static int block_begin(int nslices, int nrb, int b) { return (int)((long long)nslices * b / nrb); }

// Whether one cluster of 16 blocks of `fn` can run.
static bool cluster16(const void *fn, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = 16;
  cfg.blockDim = kResThreads;
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int nc = 0;
  const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&nc, fn, &cfg) == cudaSuccess && nc >= 1;
  if (!ok) cudaGetLastError();
  return ok;
}

// A launch shape and its block-local tables.
struct ResShape {
  int grid, nrb, k;   // form, row blocks, slices per warp of the instance
  int rows_max, halo_max, stage;
  int o[9];           // shared-memory offsets
  size_t total;       // bytes of shared memory
  std::vector<uint4> rcol;
  std::vector<int4> meta;
  std::vector<int> hptr, hids, pptr;
  std::vector<int2> push;
  std::vector<unsigned char> rle;
};

// Slices per warp of the instance for at most `k` (0: none).
static int res_k(int k, bool grid) {
  if (!grid) return k <= 1 ? 1 : k <= 2 ? 2 : 0;
  return k <= 1 ? 1 : k <= 2 ? 2 : k <= 4 ? 4 : k <= 6 ? 6 : k <= 9 ? 9 : 0;
}

// Whether the instance reads a slice of width w from shared memory wherever
// the planner has left it: kRegs' groups beyond the first.
static bool reads_resident(int k, int w) { return k <= 2 && slot_groups(w) > 1; }

// Whether behind a staged slice of width w a buffer of `groups` groups holds
// values only.  A buffer has a slice's columns and, behind them, its values,
// and slots past its end multiply what is there by zero: with slices of no or
// one slot beside others of two groups that would be column words, which may
// read as no number.  Such slices are read in place.
static bool staged_values(int w, int groups) { return 512 * slot_groups(w) + 256 * w >= 512 * groups; }

// Fills `p` for a matrix of n rows, on the host alone: `limit(k, grid, bytes)`
// gives the dynamic shared memory an instance may use, `cluster(k, bytes)`
// whether 16 of its blocks can be a cluster.  done = false where the resident
// kernel does not apply.
template <class L, class F>
static int resident_shape(int n, const JcgHostSell *h, int itmax, int nrb_req, int nsm, L limit, F cluster,
                          ResShape &p, bool &done) {
  done = false;
  const int nsl = (n + kSlice - 1) / kSlice;
  int wmax = 1;
  for (int s = 0; s < nsl; ++s) wmax = std::max(wmax, h->sl_w[s]);
  if (wmax >= 128) return ADC_OK;
  // Cluster form up to 16 blocks of two slices per warp (15,360 rows): with
  // four (24,963 rows) an iteration took 4.2 us in the cluster.  Beyond, one
  // block per SM, with at least one slice per warp.
  int grid = 1, nrb = std::max(1, std::min(nsm, (nsl + kRowWarps - 1) / kRowWarps));
  if (nrb_req > 0) nrb = std::max(1, std::min({nrb_req, nsm, nsl}));
  if (nrb_req == 0) {
    int nb = 1;
    while (nb < kMaxCluster && nb * kRowWarps < nsl) nb *= 2;
    if (nsl <= nb * kRowWarps * 2) {
      grid = 0;
      nrb = nb;
    }
  }
  int k_min = 1;
  for (;;) {   // at most three times: cluster form, grid form, grid form from k_min
    int per = 0;
    for (int b = 0; b < nrb; ++b)
      per = std::max(per, block_begin(nsl, nrb, b + 1) - block_begin(nsl, nrb, b));
    const int k = res_k(std::max(k_min, (per + kRowWarps - 1) / kRowWarps), grid != 0), rows_max = per * kSlice;
    bool fits = k != 0;
    p = ResShape();
    std::vector<uint4> &rcol = p.rcol;
    std::vector<int4> &meta = p.meta;
    std::vector<int> &hptr = p.hptr, &hids = p.hids, &pptr = p.pptr;
    std::vector<int2> &push = p.push;
    std::vector<unsigned char> &rle = p.rle;
    meta.resize(nsl);
    pptr.assign(nrb + 1, 0);
    int halo_max = 0;
    if (fits) {
      // block-local columns: a row of the block is its offset from the first
      // row, any other row rows_max + its place in the block's halo list
      size_t nvec = 0;
      for (int s = 0; s < nsl; ++s) {
        meta[s] = make_int4(h->sl_ptr[s], h->sl_w[s], (int)nvec, -1);
        nvec += slot_groups(h->sl_w[s]);
      }
      rcol.assign(std::max<size_t>(nvec * 32, 1), make_uint4(0, 0, 0, 0));
      unsigned short *lc = (unsigned short *)rcol.data();
      hptr.assign(nrb + 1, 0);
      rle.assign((size_t)nsl * kSlice, 0);
      for (int i = 0; i < n; ++i) rle[i] = (unsigned char)h->rlen[i];
      std::vector<int> stamp(n, -1), hid(n, 0), owner(nsl, 0);
      for (int b = 0; b < nrb; ++b)
        for (int s = block_begin(nsl, nrb, b); s < block_begin(nsl, nrb, b + 1); ++s) owner[s] = b;
      for (int b = 0; b < nrb; ++b) {
        const int s0 = block_begin(nsl, nrb, b), s1 = block_begin(nsl, nrb, b + 1), r0 = s0 * kSlice;
        int nh = 0;
        for (int s = s0; s < s1; ++s)
          for (int q = 0; q < 8 * slot_groups(h->sl_w[s]); ++q)
            for (int lane = 0; lane < kSlice; ++lane) {
              const int i = s * kSlice + lane;
              int l = -1;   // padding: the zero cell, set below
              if (i < n && q < h->rlen[i]) {
                const int j = h->col[(size_t)h->sl_ptr[s] + (size_t)q * kSlice + lane];
                if (j >= r0 && j < s1 * kSlice) {
                  l = j - r0;
                } else {
                  if (stamp[j] != b) {
                    stamp[j] = b;
                    hid[j] = nh++;
                    const int ob = owner[j / kSlice];
                    hids.push_back(grid ? j : (ob << 16) | (j - block_begin(nsl, nrb, ob) * kSlice));
                    rle[j] |= 128;
                  }
                  l = rows_max + hid[j];
                }
              }
              lc[((size_t)meta[s].z * 32 + (size_t)(q >> 3) * 32 + lane) * 8 + (q & 7)] = (unsigned short)l;
            }
        hptr[b + 1] = hptr[b] + nh;
        halo_max = std::max(halo_max, nh);
      }
      if (!grid) {   // the halo lists, by owner
        for (int id : hids) pptr[(id >> 16) + 1]++;
        for (int b = 0; b < nrb; ++b) pptr[b + 1] += pptr[b];
        push.resize(hids.size());
        std::vector<int> at(pptr.begin(), pptr.end() - 1);
        for (int b = 0; b < nrb; ++b)
          for (int q = hptr[b]; q < hptr[b + 1]; ++q)
            push[at[hids[q] >> 16]++] = make_int2(hids[q] & 0xffff, (b << 16) | (q - hptr[b]));
      }
      fits = rows_max + halo_max < 8191;   // byte offsets in 16 bits
      if (fits)
        for (size_t q = 0; q < nvec * 32 * 8; ++q)
          lc[q] = (unsigned short)(8 * (lc[q] == 0xffff ? rows_max + halo_max : lc[q]));
    }
    size_t total = 0;
    if (fits) {
      const size_t vb = (size_t)rows_max + halo_max + 1;   // and the zero cell
      size_t o = align_up(8 * vb, 128);
      p.o[0] = (int)o; o += align_up((grid ? 8 : 24) * (size_t)halo_max, 128);
      p.o[1] = (int)o; o += align_up(4 * (size_t)halo_max, 128);
      p.o[2] = (int)o; o += align_up(32 * (size_t)(itmax + 2), 128);
      p.o[3] = (int)o; o += align_up(16 * (size_t)per, 128);
      p.o[4] = (int)o; o += align_up(8 * (grid ? 6 : 9) * (size_t)kPart, 128);
      p.o[5] = (int)o; o += align_up(16 * kRowWarps, 128);
      int push_max = 0;
      for (int b = 0; b < nrb; ++b) push_max = std::max(push_max, pptr[b + 1] - pptr[b]);
      p.o[8] = (int)o; o += align_up(8 * (size_t)push_max, 128);
      p.o[6] = (int)o;
      size_t room_max = 0;
      if (int rc = limit(k, grid != 0, &room_max)) return rc;
      // columns and values of a slice, in whole groups of eight slots
      auto slice_bytes = [&](int w) { return (size_t)slot_groups(w) * (512 + 2048); };
      auto bytes = [&](int s) { return slice_bytes(h->sl_w[s]); };
      const size_t area0 = std::max(8 * vb, grid ? 0 : 16 * (size_t)rows_max);   // w, or exported values
      // every block's matrix beside it, or staging and what still fits
      size_t all = 0;
      for (int b = 0; b < nrb; ++b) {
        size_t t = 0;
        for (int s = block_begin(nsl, nrb, b); s < block_begin(nsl, nrb, b + 1); ++s) t += bytes(s);
        all = std::max(all, t);
      }
      size_t area = align_up(area0, 128), stage = 0, room = all;
      if (o + area + all > room_max) {
        if (!grid) {
          fits = false;
        } else {
          // staging wide enough for all but the few widest slices, which are
          // read in place
          std::vector<int> hist(wmax + 1, 0);
          for (int s = 0; s < nsl; ++s) hist[h->sl_w[s]]++;
          int wcap = wmax, over = 0;
          while (wcap > 1 && over + hist[wcap] <= nsl / 200) over += hist[wcap--];
          stage = align_up(slice_bytes(wcap), 128);
          area = align_up(std::max(area0, 2 * kRowWarps * stage), 128);
          fits = o + area <= room_max;
          room = fits ? room_max - o - area : 0;
        }
      }
      p.o[7] = (int)(o + area);
      if (fits) {
        // residency: the odd slices of every warp first, so that a streamed
        // slice's copy runs while the warp works on a resident one
        size_t used_max = 0;
        for (int b = 0; b < nrb; ++b) {
          const int s0 = block_begin(nsl, nrb, b), cnt = block_begin(nsl, nrb, b + 1) - s0;
          size_t used = 0;
          for (int pass = 0; pass < 2; ++pass)
            for (int ls = 0; ls < cnt; ++ls) {
              if (((ls / kRowWarps) & 1) != (pass == 0)) continue;
              const size_t sz = bytes(s0 + ls);
              if (used + sz <= room) {
                meta[s0 + ls].w = (int)used;
                used += sz;
              } else if (sz > stage || !staged_values(h->sl_w[s0 + ls], (int)(stage / slice_bytes(1)))) {
                meta[s0 + ls].w = -2;
              }
            }
          used_max = std::max(used_max, used);
        }
        total = o + area + used_max;
        p.stage = (int)stage;
      }
    }
    // One block per SM fits by its launch bounds and the limit above, and so
    // does a cluster of up to eight; 16 are a device's choice.
    if (fits && !grid && nrb > 8) fits = cluster(k, total);
    if (!fits) {
      if (grid) return ADC_OK;
      grid = 1;
      nrb = std::max(1, std::min(nsm, (nsl + kRowWarps - 1) / kRowWarps));
      continue;
    }
    // where shared memory ran out for slices that the instance would read
    // there, the smallest that streams them or reads them in place
    const auto misread = [k](const int4 &m) { return m.w < 0 && reads_resident(k, m.y); };
    if (std::any_of(meta.begin(), meta.end(), misread)) {
      k_min = 3;
      continue;
    }
    p.grid = grid;
    p.nrb = nrb;
    p.k = k;
    p.rows_max = rows_max;
    p.halo_max = halo_max;
    p.total = total;
    done = true;
    return ADC_OK;
  }
}

// Chooses the launch shape for a matrix, builds its block-local tables and
// uploads them; done = false where the resident kernel does not apply.
int plan_jcg_resident(adc_ctx *c, const JcgHostSell *h, int nsm, bool &done) {
  ResShape p;
  if (int rc = resident_shape(
          c->np, h, c->itmax, c->jcg_nrb_req, nsm,
          [](int k, bool grid, size_t *bytes) { return jcg_smem_limit(res_fn(k, grid), bytes); },
          [](int k, size_t bytes) { return cluster16(res_fn(k, false), bytes); }, p, done))
    return rc;
  if (!done) return ADC_OK;
  done = false;
  JcgTables T;
  const size_t o_rcol = T.add(p.rcol), o_meta = T.add(p.meta), o_hptr = T.add(p.hptr), o_hids = T.add(p.hids),
               o_rle = T.add(p.rle), o_pptr = T.add(p.pptr), o_push = T.add(p.push);
  if (int rc = T.upload(c)) return rc;
  c->jrcol = (uint4 *)(c->jtab + o_rcol);
  c->jmeta = (int4 *)(c->jtab + o_meta);
  c->jhalo_ptr = (int *)(c->jtab + o_hptr);
  c->jhalo_ids = (int *)(c->jtab + o_hids);
  c->jrle = c->jtab + o_rle;
  c->jpush_ptr = (int *)(c->jtab + o_pptr);
  c->jpush = (int2 *)(c->jtab + o_push);
  for (int q = 0; q < 9; ++q) c->jr_o[q] = p.o[q];
  c->jcg_rows_blocks = p.nrb;
  c->jcg_grid = p.nrb;
  c->jcg_res = p.grid ? 1 : 2;
  c->jcg_res_k = p.k;
  c->jcg_rows_max = p.rows_max;
  c->jcg_halo_max = p.halo_max;
  c->jcg_stage_bytes = p.stage;
  c->jcg_smem = p.total;
  done = true;
  return ADC_OK;
}

int launch_jcg_resident(const JcgArgs &a0, const adc_ctx *c) {
  JcgArgs a = a0;
  a.rows_max = c->jcg_rows_max;
  a.halo_max = c->jcg_halo_max;
  a.stage_bytes = c->jcg_stage_bytes;
  a.meta = c->jmeta;
  a.rcol = c->jrcol;
  a.rle = c->jrle;
  a.halo_ptr = c->jhalo_ptr;
  a.halo_ids = c->jhalo_ids;
  a.push_ptr = c->jpush_ptr;
  a.push = c->jpush;
  a.o_hp = c->jr_o[0]; a.o_hid = c->jr_o[1]; a.o_tri = c->jr_o[2]; a.o_meta = c->jr_o[3];
  a.o_push = c->jr_o[8];
  a.o_part = c->jr_o[4]; a.o_bar = c->jr_o[5]; a.o_area = c->jr_o[6]; a.o_res = c->jr_o[7];
  const bool grid = c->jcg_res == 1;
  const void *fn = res_fn(c->jcg_res_k, grid);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = c->jcg_rows_blocks;
  cfg.blockDim = kResThreads;
  cfg.dynamicSmemBytes = c->jcg_smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[2];
  if (grid) {
    at[0].id = cudaLaunchAttributeCooperative;   // all blocks resident: they wait for one another
    at[0].val.cooperative = 1;
    cfg.numAttrs = 1;
  } else {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c->jcg_rows_blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cfg.attrs = at;
  void *args[] = {&a};
  ADC_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  return ADC_OK;
}

}  // namespace adc

using namespace adc;

extern "C" int adc_selftest_jcg_shape(int n, const int *sl_ptr, const int *sl_w, const int *col, const int *rlen,
                                      int itmax, int row_blocks, int sms, int smem, int *out) {
  if (n < 1 || !sl_ptr || !sl_w || !col || !rlen || itmax < 0 || !out) {
    set_error("adc_selftest_jcg_shape: bad arguments");
    return ADC_ERR_ARG;
  }
  const JcgHostSell h{sl_ptr, sl_w, col, rlen};
  ResShape p;
  bool done = false;
  if (int rc = resident_shape(
          n, &h, itmax, row_blocks, sms,
          [smem](int, bool, size_t *bytes) {
            *bytes = (size_t)smem;
            return ADC_OK;
          },
          [](int, size_t) { return true; }, p, done))
    return rc;
  out[0] = !done ? 0 : p.grid ? 1 : 2;
  out[1] = done ? p.k : 0;
  out[2] = out[3] = 0;
  for (const int4 &m : p.meta)
    if (done && m.w < 0) {
      ++out[2];
      if (reads_resident(p.k, m.y)) ++out[3];
    }
  return ADC_OK;
}
