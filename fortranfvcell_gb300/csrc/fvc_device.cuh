// fvc_device.cuh -- device-side building blocks shared by the SpMV and
// Krylov kernels of libfvcgpu (sm_103a).
//
// Matrix layout on the device: sliced ELLPACK with slice height 32
// (SELL-32).  Slice s covers rows [32s, 32s+32); its width w_s is the
// longest row of the slice; entry k of lane l sits at slot
// slice_ptr[s] + 32*k + l, so one warp reads one slice with fully
// coalesced 32-bit (columns) and 64-bit (values) streams.  Padding slots
// hold column = own row and value = 0, which leaves every sum unchanged.
// Row entries keep the reference's per-row order, and the diagonal is
// applied first or last exactly where src/Matvec.f applies it, so the
// FP64 SpMV is bit-identical to the reference routine (no FMA contraction:
// products and sums are rounded separately, as the Fortran loops do).
#pragma once
#include <cooperative_groups.h>
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "fvc_internal.h"

namespace fvc {

constexpr int kSlice = 32;

template <typename V>
struct SellView {
  int n;                 // rows
  int nslices;
  const int64_t *sptr;   // nslices+1 slot offsets
  const int *col;        // 0-based columns
  const V *val;          // values (negated off-diagonals, as stored)
  const V *diag;         // n (null for DIAG_NONE)
  int diag_mode;
  const int *mirror = nullptr;  // per slot: the slot of the transposed entry
                                // (symmetric patterns; transposed solves only)
  int *chk = nullptr;           // check builds: the launch's error word
};

// Opt-in device checks (compiled with -DFVC_CHECK, the library's check
// variant; see build.py).  A column, slice width, offset or mirror index
// outside its array is recorded in an error word -- the first failing
// check's code, kept by atomicCAS -- and the access is redirected to a safe
// index (the row itself, or an empty slice), so nothing is read out of
// bounds and nothing traps.  The word is the launch's grid-wait error word:
// every grid wait sees it and returns, so the launch ends through its
// normal error path, and the host reports FVC_ERR_ARG with the check's
// name (check_status).  Without FVC_CHECK the checks compile to nothing.
enum CheckCode : int {
  kChkColumn = 101,      // SELL column outside [0, n)
  kChkSliceWidth = 102,  // slice width negative or above n
  kChkOffset = 103,      // FP32 operator: row + 16-bit offset outside [0, n)
  kChkMirror = 104,      // transposed solves: mirror slot outside the slots
  kChkCluster = 105,     // cluster PCG: a column whose owner CTA is not in the cluster
};
#ifdef FVC_CHECK
#define FVC_CHK(cond, word, code, fix)                        \
  do {                                                        \
    if (!(cond)) {                                            \
      int *w_ = (word);                                       \
      if (w_) atomicCAS(w_, 0, (int)(code));                  \
      fix;                                                    \
    }                                                         \
  } while (0)
#else
#define FVC_CHK(cond, word, code, fix) \
  do {                                 \
  } while (0)
#endif

// One block's partial of one reduced quantity with the episode that wrote
// it, moved by single 16-byte accesses: a reader that finds the episode has
// the value, with no ordering between the slot and any other word.
struct __align__(16) RedSlot {
  unsigned long long v, ep;
};

// Grid synchronisation state of one persistent launch.  `count` is a
// monotonically increasing arrival counter (episode e completes when it
// reaches e * nblocks, so it never needs resetting inside the launch).  The
// slots rotate over four sets so a block running ahead never overwrites
// data still read; they are zeroed with the counter before the launch, so
// that no slot carries an episode of an earlier one.
struct GridSync {
  unsigned int *count;     // [0] arrivals of the sums and barriers; [8] (its
                           // own 32-byte sector) publications (exchange_totals)
  unsigned long long *xw;  // words of the exact sums (exact_sum)
  int *err;                // sticky error (FVC_ERR_TIMEOUT on a stuck wait)
  RedSlot *slots;          // 4 sets x kMaxNV x nblocks
  unsigned int nblocks;    // blocks that synchronise through this state
  unsigned int base;       // blockIdx.x of the first of them (0 for a whole grid)
  // nonzero: the nblocks blocks are one thread-block cluster; the waits
  // and reductions below then use the cluster barrier and distributed
  // shared memory instead of global memory (cluster_exchange)
  int cluster = 0;
};

// How often this launch has synchronised: reductions and barriers (the
// episodes of the counter and the slots), published, and summed exactly.
struct Episode {
  unsigned int n = 0, pub = 0, x = 0;
};

constexpr int kMaxNV = 4;

// The cluster form of a reduction.  Lane 0 of warp 0 of every CTA has
// stored its block's NV partials in its own slot; every thread of every CTA
// has then met at the cluster barrier (arrive.release / wait.acquire at
// cluster scope: the slots, and every global-memory write made before it,
// are visible to the whole cluster after it).  Here warp 0 reads
// the CTAs' slots in rank order through distributed shared memory and sums
// them in a fixed shuffle tree, so every CTA holds identical totals (in lane
// 0 of warp 0).  There is no spin-wait: the barrier is the hardware's, and
// every CTA reaches it the same number of times because every branch
// around it depends only on those identical totals.  Two slots alternate
// (a slot is written again only after a later barrier, so never while a
// CTA still reads it), and the kernel ends with one more barrier so that
// no CTA's shared memory goes away while another reads it.
template <int NV>
__device__ __forceinline__ void cluster_exchange(double (*slots)[kMaxNV], unsigned int ep,
                                                 double (&t)[NV]) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int nb = (int)cl.num_blocks();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double u = (lane < nb) ? *cl.map_shared_rank(&slots[ep & 1u][q], lane) : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)  // at most 16 CTAs
        u = __dadd_rn(u, __shfl_down_sync(0xffffffffu, u, o));
      t[q] = u;
    }
  }
}

// the closing barrier of a kernel whose blocks reduce through cluster_exchange
__device__ __forceinline__ void cluster_close(const GridSync &gs) {
  if (gs.cluster) cooperative_groups::this_cluster().sync();
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void red_add_release(unsigned int *p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_relaxed(unsigned int *p, unsigned int v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_slot(RedSlot *p, double v, unsigned int ep) {
  asm volatile(
      "{\n .reg .b128 r;\n mov.b128 r, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], r;\n}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"((unsigned long long)ep)
      : "memory");
}
__device__ __forceinline__ RedSlot ld_slot(const RedSlot *p) {
  RedSlot s;
  asm volatile(
      "{\n .reg .b128 r;\n ld.relaxed.gpu.global.b128 r, [%2];\n mov.b128 {%0, %1}, r;\n}"
      : "=l"(s.v), "=l"(s.ep)
      : "l"(p)
      : "memory");
  return s;
}

// Every wait is bounded: after kBarrierTimeoutNs the block records
// FVC_ERR_TIMEOUT and leaves; the other waiters see the flag and leave too,
// so a broken launch returns an error instead of spinning.
constexpr uint64_t kBarrierTimeoutNs = 4000000000ull;  // 4 s

// Waits until count reaches target; called by a whole warp.  kAcquire: what
// the other blocks wrote before their release arrivals is visible afterwards.
// All lanes poll, with a vote per turn: after a spin loop that a part of a
// warp ran, the warp went on in pieces -- __syncwarp or not -- and a chain of
// shuffles and FP64 additions took 2830 instead of 670 clocks.  The error word
// and the clock are looked at every 64th poll only: in every poll they cost
// another trip to L2 and delayed the hit by half of it.  False, with err set,
// when the wait exceeded its bound.
template <bool kAcquire>
__device__ __forceinline__ bool wait_count(const unsigned int *count, int *err,
                                           unsigned int target) {
  unsigned int spins = 0;
  uint64_t t0 = 0;
  bool ok = true;
  while (__any_sync(0xffffffffu,
                    (kAcquire ? ld_acquire(count) : ld_relaxed(count)) < target)) {
    if ((++spins & 63u) == 0) {
      const uint64_t now = global_ns();
      if (t0 == 0) t0 = now;
      const bool late = now - t0 > kBarrierTimeoutNs;
      if (__any_sync(0xffffffffu, late || *(volatile int *)err != 0)) {
        if (late) atomicExch(err, 7 /* FVC_ERR_TIMEOUT */);
        ok = false;
        break;
      }
    }
  }
  return ok;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum of NV values per thread; result valid in thread 0.
// Fixed tree order -> deterministic.  red must hold NV*32 doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) red[q * 32 + warp] = v[q];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double t = (lane < nwarps) ? red[q * 32 + lane] : 0.0;
      v[q] = warp_sum(t);
    }
  }
  __syncthreads();
}

// The partials of one quantity summed in block order (lane l takes blocks
// l, l + 32, ...): the same total in every block, valid in lane 0.  The
// slots must hold their values (an acquire wait on count).
__device__ __forceinline__ double sum_slots(const RedSlot *p, unsigned int nb) {
  const unsigned int lane = threadIdx.x & 31;
  double t = 0.0;
#pragma unroll 1
  for (unsigned int b = lane; b < nb; b += 32)
    t = __dadd_rn(t, __longlong_as_double((long long)ld_slot(p + b).v));
  return warp_sum(t);
}

// Grid-wide barrier that publishes every block's writes: one release
// arrival per block, one acquire poll of the counter.  Returns false, with
// gs.err set, when the wait exceeded its bound.
__device__ __forceinline__ bool grid_barrier(const GridSync &gs, Episode &episode) {
  __shared__ int s_ok;
  __syncthreads();
  const unsigned int ep = ++episode.n;
  if (gs.cluster) {
    cooperative_groups::this_cluster().sync();
    return true;
  }
  if (gs.nblocks == 1) return true;
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) red_add_release(gs.count, 1u);
    const bool ok = wait_count<true>(gs.count, gs.err, ep * gs.nblocks);
    if (threadIdx.x == 0) s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  return s_ok != 0;
}

// Deterministic all-reduce of NV doubles per thread, publishing the blocks'
// writes like grid_barrier: every block sums the partials itself in block
// order.  The totals are in every thread's v.
template <int NV>
__device__ __forceinline__ bool grid_allreduce(const GridSync &gs, Episode &episode,
                                               double (&v)[NV], double *red) {
  __shared__ int s_ok;
  block_sum<NV>(v, red);
  const unsigned int ep = ++episode.n;
  if (gs.cluster) {
    __shared__ double s_slot[2][kMaxNV];
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q) s_slot[ep & 1u][q] = v[q];
    double t[NV];
    cooperative_groups::this_cluster().sync();
    cluster_exchange<NV>(s_slot, ep, t);
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q) red[q] = t[q];
  } else if (gs.nblocks == 1) {  // one block: its sum is the total (same value)
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q) red[q] = v[q];
  } else {
    const unsigned int nb = gs.nblocks;
    RedSlot *part = gs.slots + (size_t)(ep & 3u) * kMaxNV * nb;
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q)
          st_slot(part + (size_t)q * nb + (blockIdx.x - gs.base), v[q], ep);
        red_add_release(gs.count, 1u);
      }
      const bool ok = wait_count<true>(gs.count, gs.err, ep * nb);
      if (threadIdx.x == 0) s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    if (!s_ok) return false;
    const int warp = threadIdx.x >> 5;
    if (warp < NV) {
      const double t = sum_slots(part + (size_t)warp * nb, nb);
      if ((threadIdx.x & 31) == 0) red[warp] = t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = red[q];
  __syncthreads();
  return true;
}

// The exchange of the grid-wide sums of the mixed-precision CG
// (grid_allreduce_ff) and of grid_allreduce.  Thread 0 puts its block's partial of each quantity
// into its slots and counts itself in; every block then waits for all and
// sums all partials itself in a fixed order, so that every block holds
// identical totals.
//
// The arrival is relaxed, so that it does not wait for the block's stores to
// be performed, and each partial carries its episode, so the slots need no
// ordering against the counter (a slot read too early is read again); 152
// blocks: 2.12 instead of 2.97 us for one double with 128 threads, 2.74
// instead of 3.62 us with 1024, against a release arrival and an acquire
// wait.  Polling the slots alone, without the counter, took 3.8 us: 152
// blocks reading 2.4 KB over and over keep the writers off the same lines.
template <int NV>
__device__ __forceinline__ void grid_arrive(const GridSync &gs, unsigned int ep,
                                            const double (&bsum)[NV]) {
  const unsigned int nb = gs.nblocks;
  RedSlot *part = gs.slots + (size_t)(ep & 3u) * kMaxNV * nb + (blockIdx.x - gs.base);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_slot(part + (size_t)q * nb, bsum[q], ep);
  red_add_relaxed(gs.count, 1u);
}

// The partials of cnt blocks from slot i0 on into out (shared memory): the
// whole block, one slot per thread.  (A lane's five slots held together cost the
// solvers' loops spills, and the staged kernels, whose shared memory leaves no
// L1, a third of their speed.)
__device__ __forceinline__ void read_slots(const GridSync &gs, unsigned int ep, unsigned int i0,
                                           unsigned int cnt, double *out) {
  const RedSlot *p = gs.slots + (size_t)(ep & 3u) * kMaxNV * gs.nblocks + i0;
  const unsigned int lane = threadIdx.x & 31u;
#pragma unroll 1
  for (unsigned int w = threadIdx.x - lane; w < cnt; w += blockDim.x) {
    const unsigned int i = min(w + lane, cnt - 1);
    RedSlot s = ld_slot(p + i);
    unsigned int tries = 0;
    // (the counter passed a slot's store: read again)
    while (__any_sync(0xffffffffu, s.ep != ep)) {
      if (++tries == (1u << 24)) {  // (seconds; a store takes none)
        atomicExch(gs.err, 7 /* FVC_ERR_TIMEOUT */);
        break;
      }
      s = ld_slot(p + i);
    }
    if (w + lane < cnt) out[i] = __longlong_as_double((long long)s.v);
  }
}

// The cluster barrier with mid() run by thread 0 between its arrival and its
// wait (what it costs hides in the barrier's latency).
template <typename M>
__device__ __forceinline__ void cluster_sync_mid(M &&mid) {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  if (threadIdx.x == 0) mid();
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The last step of both sums: thread 0 holds its block's partials.
// kPublish: the blocks' vector writes before it are visible to the other
// blocks after it, for a next phase that gathers them.  A second counter
// carries that (release arrival and acquire wait of warp 2), beside the
// partials and not before them: its wait for the block's stores hides in the
// sum's two trips to L2.  tot: shared memory for cap partials of each quantity.
// overlap(): work of the warps that take no part, while the others wait.
struct NoOverlap {
  __device__ void operator()() const {}
};
template <int NV, bool kPublish, typename S, typename M, typename F, typename O = NoOverlap>
__device__ __forceinline__ bool exchange_totals(const GridSync &gs, Episode &episode,
                                                const double (&bsum)[NV], double *tot,
                                                unsigned int cap, S &&side, M &&mid, F &&f,
                                                O &&overlap = O()) {
  __shared__ int s_ok[2];
  __shared__ double s_t[NV];
  if (kPublish) ++episode.pub;
  const unsigned int ep = ++episode.n;
  if (gs.nblocks == 1) {  // one block: its sum is the total (same value)
    if (threadIdx.x == 0) {
      mid();
      f(bsum);
    } else if (threadIdx.x == 32) {
      side();
    } else if (threadIdx.x >= 96) {
      overlap();
    }
    __syncthreads();
    return true;
  }
  const unsigned int nb = gs.nblocks;
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      grid_arrive<NV>(gs, ep, bsum);
      mid();
    }
    const bool ok = wait_count<false>(gs.count, gs.err, ep * nb);
    if (threadIdx.x == 0) s_ok[0] = ok ? 1 : 0;
  } else if (threadIdx.x < 64) {
    if (threadIdx.x == 32) side();
  } else if (kPublish && threadIdx.x < 96) {
    if (threadIdx.x == 64) red_add_release(gs.count + 8, 1u);
    const bool ok = wait_count<true>(gs.count + 8, gs.err, episode.pub * nb);
    if (threadIdx.x == 64) s_ok[1] = ok ? 1 : 0;
  } else if (threadIdx.x >= 96) {
    overlap();
  }
  __syncthreads();
  if (!s_ok[0] || (kPublish && !s_ok[1])) return false;
  // the partials of quantity q in block order: lane l of warp q takes blocks
  // l, l + 32, ... (from shared memory, cap at a time)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double u = 0.0;
#pragma unroll 1
  for (unsigned int b0 = 0; b0 < nb; b0 += cap) {
    const unsigned int cnt = min(nb - b0, cap);
#pragma unroll
    for (int q = 0; q < NV; ++q) read_slots(gs, ep, q * nb + b0, cnt, tot + q * cap);
    __syncthreads();
    if (warp < NV) {
      const double *p = tot + warp * cap;
#pragma unroll 1
      for (unsigned int b = lane; b < cnt; b += 128) {
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (b + 32 * k < cnt) ? p[b + 32 * k] : 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (b + 32 * k < cnt) u = (b0 == 0 && b < 32 && k == 0) ? v[0] : __dadd_rn(u, v[k]);
      }
    }
    if (b0 + cap < nb) __syncthreads();  // before tot is filled again
  }
  if (warp < NV) {
    u = warp_sum(u);
    if (lane == 0) s_t[warp] = u;
  }
  if (NV > 1) __syncthreads();
  if (threadIdx.x == 0) f(s_t);
  __syncthreads();
  return true;
}

// A block's sum of NV FP64 values per thread in a fixed order, in lane 0 of warp
// 0: four warps add blockDim / 128 values per lane (buf: NV x blockDim doubles;
// blockDim.x a multiple of 128), warp 0 adds the four per lane and finishes with
// a shuffle tree.
template <int NV>
__device__ __forceinline__ void ordered_block_sum(const double (&v)[NV], double *buf,
                                                  double (&t)[NV]) {
  __shared__ double s_part[NV][128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bd = blockDim.x, per = bd >> 7;  // values per lane of the first level
#pragma unroll
  for (int q = 0; q < NV; ++q) buf[q * bd + threadIdx.x] = v[q];
  __syncthreads();
  if (warp < 4) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const double *b = buf + q * bd + warp * (bd >> 2) + lane;
      double u = b[0];
      for (int k = 1; k < per; ++k) u = __dadd_rn(u, b[32 * k]);
      s_part[q][threadIdx.x] = u;
    }
  }
  __syncthreads();
  if (warp == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double u = s_part[q][lane];
#pragma unroll
      for (int k = 1; k < 4; ++k) u = __dadd_rn(u, s_part[q][32 * k + lane]);
      t[q] = warp_sum(u);
    }
}

// Sums in that order: over one cluster or block, the CTAs following in rank
// order (the cluster BiCGSTAB, see Scratch::ordered), or over a grid, the blocks
// in block order (exchange_totals; the PCG of kOrderedRows rows and more).
// Thread 0 then calls f(totals) -- the place for the iteration's scalar FP64
// work -- and one __syncthreads hands its results (through shared memory) to
// the block.  Scalar work that needs nothing of this sum (a division is 570
// clocks) hides in the wait: thread 0 calls mid() between its arrival and its
// wait, for values f uses; thread 32 calls side(), for values of later phases;
// over a grid the warps from the fourth on run overlap().
template <int NV, typename S, typename M, typename F>
__device__ __forceinline__ void ordered_sum(const GridSync &gs, Episode &episode,
                                            const double (&v)[NV], double *buf, S &&side, M &&mid,
                                            F &&f) {
  __shared__ double s_slot[2][kMaxNV];
  double t[NV];
  ordered_block_sum<NV>(v, buf, t);
  const unsigned int ep = ++episode.n;
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) s_slot[ep & 1u][q] = t[q];
  if (threadIdx.x == 32) side();
  __syncwarp();
  if (gs.cluster) {
    cluster_sync_mid(mid);
    cluster_exchange<NV>(s_slot, ep, t);
  } else if (threadIdx.x == 0) {
    mid();
  }
  if (threadIdx.x == 0) f(t);
  __syncthreads();
}
template <int NV, bool kPublish, typename S, typename M, typename F, typename O>
__device__ __forceinline__ bool ordered_grid_sum(const GridSync &gs, Episode &episode,
                                                 const double (&v)[NV], double *buf, S &&side,
                                                 M &&mid, F &&f, O &&overlap) {
  double t[NV];
  ordered_block_sum<NV>(v, buf, t);
  return exchange_totals<NV, kPublish>(gs, episode, t, buf, blockDim.x, side, mid, f, overlap);
}

// ---- scalar work of the recurrences ---------------------------------------
// One thread does it between two phases, so its dependent FP64 instructions
// (64 clocks each; a division 570, a square root 570) are the whole grid's
// wait.

// (Functions: their callers are one thread's code between two phases.)
static __device__ __noinline__ double divide(double t, double d) { return t / d; }
static __device__ __noinline__ double root(double v) { return sqrt(v); }

__device__ __forceinline__ bool not_finite_bits(double v) {
  return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}

// A divisor whose reciprocal was taken ahead of the dividend.
struct Divisor {
  double d, r;  // r = 1/d, or 0 when d is too far from 1 for quotient()
  __device__ __forceinline__ void set(double v) {
    d = v;
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    r = (e > 1023 - 500 && e < 1023 + 500) ? divide(1.0, v) : 0.0;
  }
};

// t / d by Markstein's correction of t * (1/d) (IBM J. Res. Dev. 34, 1990):
// three dependent FMAs after t instead of a division; within half an ulp and
// a few parts in 2^53 of it.  Divisors out of range, and quotients that are
// not finite, take the division.
__device__ __forceinline__ double quotient(double t, const Divisor &v) {
  const double q = t * v.r;
  const double z = fma(fma(-q, v.d, t), v.r, q);
  if (__double_as_longlong(v.r) == 0 || (__double2hiint(z) & 0x7ff00000) == 0x7ff00000)
    return divide(t, v.d);
  return z;
}

// t / d from scratch: the reciprocal's hardware approximation (rcp.approx.f64,
// 20 bits and more) r, one Newton step for it and for t r side by side,
// Markstein's correction as above (about 300 clocks against 570 of the
// division).  Divisors out of range, and
// quotients that are not finite, take the division.
__device__ __forceinline__ double quick_quotient(double t, double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double h = fma(-d, r, 1.0), q0 = t * r;
  r = fma(h, r, r);
  const double q = fma(h, q0, q0);
  const double z = fma(fma(-q, d, t), r, q);
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  if (e <= 1023 - 500 || e >= 1023 + 500 || not_finite_bits(z)) return divide(t, d);
  return z;
}

// The stopping test sqrt(s) < conv, without the square root while s is
// clearly above conv^2 (bound from sqrt_bound; s >= 0 or NaN: the bits of
// nonnegative doubles order like the numbers, a NaN above all of them).
__device__ __forceinline__ long long sqrt_bound(double conv) {
  const double c2 = conv * conv;
  // conv^2 not a normal number: always take the square root
  if (!(c2 > 1.0e-290 && c2 < 1.0e290)) return 0x7ff0000000000000ll;
  return __double_as_longlong(c2 * (1.0 + 1.0e-14));
}
__device__ __forceinline__ bool sqrt_below(double s, double conv, long long bound) {
  if (__double_as_longlong(s) > bound) return false;
  return root(s) < conv;
}
__device__ __forceinline__ bool is_nan_bits(double v) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

// No scalar work beside a sum.
struct NoScalars {
  __device__ void operator()() const {}
};

// ---- exact sums --------------------------------------------------------------
// The sums above cost a chain of some 25 dependent FP64 additions (64 clocks
// each) and the reading of every block's partial; at 66k rows the two sums of
// a CG iteration were two thirds of it.  The sums below add integers instead.
// Every thread splits its FP64 partial into kLimbs signed limbs of kLimbBits
// bits of one fixed-point window that all blocks know (its top lies
// kWindowHead bits above the total of the same sum one iteration ago); a
// warp adds a limb with one redux, the warps of a block theirs in shared
// memory by atomics (a second redux over the warps took 330 clocks, this 60),
// and the blocks into one 64-bit word per limb with relaxed atomics.
// Integer addition is associative, so the total does not depend on the
// order: deterministic, and exact but for the bits below the window (less
// than 2^-53.7 of the total, see sum_bad), rounded once.  The word's upper bits
// count the blocks that have added, so that one poll of the words is the whole
// exchange: no slots, no counter, no order between them.  The words only
// grow; a total is the difference to their value one use earlier (snap).
//
// A sum whose window does not hold it -- a partial at or above its top (or
// NaN, Inf), or a total that has dropped by more than 2^22, the same verdict
// in every block -- is taken again in a window set by the largest partial of
// all blocks (window_by_partials), as is the first of a kind.
//
constexpr int kLimbs = 6, kLimbBits = 21, kWindowBits = kLimbs * kLimbBits, kWindowHead = 32;
// Words of one set (two sets alternate): limb k of quantity q at 8 q + k, so
// that the atomics of a block, and each poll of it, are one request.  With a
// line of 128 bytes per word the polls of 152 blocks queued at the L2 slices
// that held two of the words: sums of 4 thousand clocks became 9, depending on
// the buffer's address.
constexpr int kXWords = 32;
constexpr int kNoWindow = INT_MIN;
constexpr int kXBlocks = 2047;            // most blocks a word's count serves

// A block's state of the exact sums (shared memory).
struct ExactState {
  unsigned long long snap[2][kXWords];
  // the block's sums (two sets alternate, all zero between uses): limb k of
  // quantity q at 8 q + k, the warps with a value above the window at 8 q + 6
  int acc[2][32];
  int flag, pub_ok;
  int nan;  // some partial was NaN or Inf: so is the total
};
// The window of one kind of sum: its top, an exponent of two, per quantity.
template <int NV>
struct SumWindow {
  int top[NV];
};

__device__ __forceinline__ int window_top(double total) {
  const int e = (__double2hiint(total) >> 20) & 0x7ff;
  // zero, subnormal, NaN or Inf: none.  (Near the ends of the exponents a window is as
  // good as elsewhere: below the smallest subnormal there is nothing to drop.)
  return (e == 0 || e == 0x7ff) ? kNoWindow : e - 1022 + kWindowHead;
}
template <int NV>
__device__ __forceinline__ void window_set(SumWindow<NV> &w, const double *t) {
#pragma unroll
  for (int q = 0; q < NV; ++q) w.top[q] = window_top(t[q]);
}

// A warp's values +-m 2^e (m < 2^kMant; up to two per lane) as limbs of the window
// with the given top, added over the warp and then to the block's acc[k] for
// limb k.  True in the lanes whose value does not fit.
template <int kMant>
__device__ __forceinline__ bool add_limbs(int (&l)[kLimbs], unsigned long long m, int e, int neg,
                                          int top) {
  const int s = e - (top - kWindowBits);  // bit of the window m starts at
  unsigned long long hi = 0, lo;
  if (s >= 64) {
    lo = 0;
    hi = m << (s & 63);
  } else if (s > 0) {
    lo = m << s;
    hi = m >> (64 - s);
  } else {
    lo = (s > -64) ? m >> -s : 0;
  }
  constexpr int M = (1 << kLimbBits) - 1;
  const int x[kLimbs] = {(int)lo & M,
                         (int)(lo >> 21) & M,
                         (int)(lo >> 42) & M,
                         (int)((lo >> 63) | (hi << 1)) & M,
                         (int)(hi >> 20) & M,
                         (int)(hi >> 41) & M};
#pragma unroll
  for (int k = 0; k < kLimbs; ++k) l[k] += (x[k] ^ -neg) + neg;
  // (with the bound of FP64, FP32 parts lost 29 of the kWindowHead bits: up to every
  // third sum of a BiCGSTAB whose products cancel was taken again)
  return s > kWindowBits - kMant - 1;
}
__device__ __forceinline__ void warp_limbs(const int (&l)[kLimbs], bool ovf, int *acc) {
  const int lane = threadIdx.x & 31;
  int mine = __any_sync(0xffffffffu, ovf) ? 1 : 0;  // lane kLimbs
#pragma unroll
  for (int k = 0; k < kLimbs; ++k) {
    const int r = __reduce_add_sync(0xffffffffu, l[k]);
    if (lane == k) mine = r;
  }
  if (lane <= kLimbs) atomicAdd(acc + lane, mine);
}
__device__ __forceinline__ void put_limbs(double v, int top, int *acc) {
  int l[kLimbs] = {0, 0, 0, 0, 0, 0};
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int ex = (int)(b >> 52) & 0x7ff;
  const unsigned long long m = (b & 0xfffffffffffffull) | ((unsigned long long)(ex != 0) << 52);
  const bool ovf = add_limbs<53>(l, m, (ex ? ex : 1) - 1075, (int)(b >> 63), top);
  warp_limbs(l, ovf, acc);
}
// The value of an FP32 pair, its parts renormalised so that they do not overlap
__device__ __forceinline__ void put_limbs(float s, float c, int top, int *acc) {
  int l[kLimbs] = {0, 0, 0, 0, 0, 0};
  const float hi = __fadd_rn(s, c);
  const float lo = __fsub_rn(c, __fsub_rn(hi, s));
  bool ovf = false;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const unsigned int b = __float_as_uint(k ? lo : hi);
    const int ex = (int)(b >> 23) & 0xff;
    const unsigned int m = (b & 0x7fffffu) | ((unsigned int)(ex != 0) << 23);
    // NaN and Inf: an exponent no window holds
    const int e = ex == 0xff ? 4096 : (ex ? ex : 1) - 150;
    ovf = add_limbs<24>(l, (unsigned long long)m, e, (int)(b >> 31), top) || ovf;
  }
  warp_limbs(l, ovf, acc);
}

// m 2^(e - 1086) (m's top bit set, rest: something below it), e < 1, as the bits of
// a subnormal, rounded to nearest even.  Cold.
static __device__ __noinline__ unsigned long long subnormal_bits(unsigned long long m, bool rest,
                                                                 int e) {
  const int sh = 12 - e;  // below the last bit
  if (sh > 64) return 0;
  unsigned long long r = sh < 64 ? m >> sh : 0;
  const unsigned long long rem = m << (64 - sh), half = 1ull << 63;
  r += (rem > half || (rem == half && (rest || (r & 1)))) ? 1 : 0;
  return r;
}
// T units of the window (its top) in FP64, rounded to nearest even (Inf above its
// exponents).  All in integers: a conversion and an FP64
// addition are 60 clocks and more of the sum's critical path each.
__device__ __forceinline__ double window_value(__int128 T, int top) {
  const bool neg = T < 0;
  const unsigned __int128 U = neg ? -(unsigned __int128)T : (unsigned __int128)T;
  const unsigned long long h = (unsigned long long)(U >> 64), l = (unsigned long long)U;
  const unsigned long long a = h ? h : l, b = h ? l : 0;
  const int z = __clzll((long long)a);
  const unsigned long long m = (a << z) | ((b >> 1) >> (63 - z)), rest = b << z;
  const unsigned int rem = (unsigned int)m & 0x7ffu;
  unsigned long long r = m >> 11;
  r += (rem > 0x400u || (rem == 0x400u && (rest != 0 || (r & 1)))) ? 1 : 0;
  const int e = top - kWindowBits + (h ? 127 : 63) - z + 1023;
  unsigned long long v = ((unsigned long long)(e - 1) << 52) + r;
  if (e >= 0x7ff) v = 0x7ff0000000000000ull;
  if (a == 0)
    v = 0;
  else if (e <= 0)
    v = subnormal_bits(m, rest != 0, e);
  return __longlong_as_double((long long)(v | ((unsigned long long)neg << 63)));
}
// Whether a total lies so low in its window that what the threads dropped
// below it (up to 2^18.3 threads, less than one unit each) could matter:
// below 2^72 units.
__device__ __forceinline__ bool sum_bad(double t, int top) {
  const int e = ((__double2hiint(t) >> 20) & 0x7ff) - 1023;
  return e < top - kWindowBits + 72;
}

__device__ __forceinline__ void exact_init(ExactState &xs) {  // a __syncthreads must follow
#pragma unroll 1
  for (int i = threadIdx.x; i < 2 * kXWords; i += blockDim.x) {
    (&xs.snap[0][0])[i] = 0;
    (&xs.acc[0][0])[i] = 0;
  }
}

// The top of a window that holds partials of biased exponents up to m and the
// sum of 2^19 of them
__device__ __forceinline__ int top_of_partials(int m) {
  return max(min(m, 0x7fe), 1) - 1022 + 1 + 19;
}

// The window of a sum from its partials: its top above the largest exponent
// (ex, biased) of all threads of all blocks, by a maximum exchanged through
// the reduction slots and a barrier.  Cold: the first sum of a kind, and one
// that its window did not hold.  False when a wait exceeded its bound.
// All by value: a reference to gs kept its owner (a batch kernel's whole MArgs, 416
// bytes) in local memory for the length of the solve (batches 1-6 % slower).
static __device__ __noinline__ bool window_by_partials(RedSlot *slots, unsigned int *count,
                                                       int *err, unsigned int nb, unsigned int me,
                                                       int cluster, unsigned int ep,
                                                       ExactState &xs, int *top, int nv, int ex0,
                                                       int ex1, int ex2, int *part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __shared__ int s_ok;
  slots += (size_t)(ep & 3u) * kMaxNV * nb;
  __syncthreads();  // part is free
  for (int q = 0; q < nv; ++q) {
    const int m = __reduce_max_sync(0xffffffffu, q == 0 ? ex0 : q == 1 ? ex1 : ex2);
    if (lane == 0) part[q * 32 + warp] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < nv; ++q) {
      int m = 0;
      for (int w = 0; w < nw; ++w) m = max(m, part[q * 32 + w]);
      st_slot(slots + (size_t)q * nb + me, (double)m, ep);
    }
    // (one block and a cluster count no arrivals, see grid_barrier)
    if (nb > 1 && !cluster) red_add_release(count, 1u);
  }
  if (cluster) cooperative_groups::this_cluster().sync();
  if (warp == 0) {
    const bool ok =
        nb == 1 || cluster || wait_count<true>(count, err, ep * nb);
    if (lane == 0) s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  if (!s_ok) return false;
  if (warp == 0) {
    bool nan = false;
    for (int q = 0; q < nv; ++q) {
      int m = 0;
      for (unsigned int b = lane; b < nb; b += 32)
        m = max(m, (int)__longlong_as_double((long long)ld_slot(slots + (size_t)q * nb + b).v));
      m = __reduce_max_sync(0xffffffffu, m);
      nan = nan || m == 0x7ff;
      if (lane == 0) top[q] = top_of_partials(m);
    }
    if (lane == 0) xs.nan = nan ? 1 : 0;
  }
  __syncthreads();
  return true;
}

// Warp 0's part of an exact sum.  First the block's limbs: lane 8 q + k gets
// limb k of quantity q with the overflow mark in bits 42 on; acc is zero again.
__device__ __forceinline__ long long block_limbs(int *acc) {
  const int lane = threadIdx.x & 31;
  const int w = acc[lane];
  acc[lane] = 0;
  const bool o = __any_sync(0xffffffffu, (lane & 7) == kLimbs && w != 0);
  return ((lane & 7) < kLimbs ? w : 0) + ((long long)(o ? 1 : 0) << 42);
}
// Then, from the limbs of all blocks (L, |L| < 2^41) and whether any overflowed
// (bad), the totals t (in every lane), each rounded once, and the verdict: 0 a
// wait exceeded its bound, 1 good, 2 the window did not hold it (never where
// it follows from the partials, sure: it has room for the sum of all threads).
template <int NV>
__device__ __forceinline__ int limb_totals(long long L, bool bad, bool ok, bool sure,
                                           const SumWindow<NV> &win, const ExactState &xs,
                                           double (&t)[NV]) {
  const int lane = threadIdx.x & 31, lq = lane >> 3, lk = lane & 7;
  const bool mine = lq < NV && lk < kLimbs;
  const int top = win.top[lq < NV ? lq : 0];
  L += __shfl_down_sync(0xffffffffu, L, 1) << kLimbBits;
  const int l0 = lane & 24;
  const long long p0 = __shfl_sync(0xffffffffu, L, l0);
  const long long p1 = __shfl_sync(0xffffffffu, L, l0 + 2);
  const long long p2 = __shfl_sync(0xffffffffu, L, l0 + 4);
  double tq = window_value(
      (__int128)p0 + ((__int128)p1 << (2 * kLimbBits)) + ((__int128)p2 << (4 * kLimbBits)), top);
  if (sure) {
    bad = false;  // only NaN and Inf overflow such a window
    if (xs.nan) tq = __longlong_as_double(0x7ff8000000000000ll);
  } else {  // (2^42 of the highest pair: the next doubling leaves 128 bits)
    bad = mine && (bad || sum_bad(tq, top) ||
                   (unsigned long long)(p2 + (1ll << 42)) >= (1ull << 43));
  }
  bad = __any_sync(0xffffffffu, bad);
  ok = __all_sync(0xffffffffu, ok);
#pragma unroll
  for (int q = 0; q < NV; ++q) t[q] = __shfl_sync(0xffffffffu, tq, 8 * q);
  return !ok ? 0 : bad ? 2 : 1;
}
// The exchange over a grid between the two, through the words of this set.
template <int NV>
__device__ __forceinline__ int exact_words(unsigned long long *xw, int *err, unsigned int nb,
                                           unsigned int set, bool sure, const SumWindow<NV> &win,
                                           ExactState &xs, double (&t)[NV]) {
  const int lane = threadIdx.x & 31, lq = lane >> 3, lk = lane & 7;
  const bool mine = lq < NV && lk < kLimbs;
  const long long w = block_limbs(xs.acc[set]);
  long long L = 0;
  bool ok = true, bad = false;
  if (nb == 1) {  // its limbs are the total
    L = (long long)((unsigned long long)w << 22) >> 22;
    return limb_totals<NV>(L, w != L, true, sure, win, xs, t);
  }
  // (the other lanes poll along on the first word, see wait_count)
  unsigned long long *word = xw + set * kXWords + (mine ? lane : 0);
  if (mine)  // bits 0-41 the limb, 42-52 blocks that overflowed, 53-63 blocks
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(w + (1ll << 53))
                 : "memory");
  const unsigned long long prev = xs.snap[set][mine ? lane : 0];
  __syncwarp();
  unsigned long long now;
  unsigned int spins = 0;
  uint64_t t0 = 0;
  for (;;) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(word) : "memory");
    const long long d = (long long)(now - prev);
    L = (long long)((unsigned long long)d << 22) >> 22;
    const unsigned int c = (unsigned int)((unsigned long long)(d - L) >> 42);
    bad = (c & 2047u) != 0;
    if (__all_sync(0xffffffffu, (c >> 11) == nb)) break;
    if ((++spins & 63u) == 0) {
      const uint64_t ns = global_ns();
      if (t0 == 0) t0 = ns;
      const bool late = ns - t0 > kBarrierTimeoutNs;
      if (__any_sync(0xffffffffu, late || *(volatile int *)err != 0)) {
        if (late) atomicExch(err, 7 /* FVC_ERR_TIMEOUT */);
        ok = false;
        break;
      }
    }
  }
  if (mine) xs.snap[set][lane] = now;
  return limb_totals<NV>(L, bad, ok, sure, win, xs, t);
}

// Warps 0 and 1 of the block meet (the values of side() for f()).
__device__ __forceinline__ void join_warps01() {
  __syncwarp();
  asm volatile("barrier.sync 1, 64;" ::: "memory");
}

// Grid-wide deterministic sum of NV values per thread: put(q, top, acc) adds
// the limbs of the warp's values of quantity q (put_limbs), expo(q) gives the
// value's biased FP64 exponent.  part: shared memory for NV * 32 ints.  win: the window of this kind of sum.  Thread 0 calls f(totals) as in
// ordered_sum; thread 32 calls side() while warp 0 exchanges (kJoin: for values
// f uses); the warps from the fourth on run overlap() meanwhile.  kPublish: as
// in exchange_totals.  Returns false when a wait
// exceeded its bound (gs.err set).
template <int NV, bool kPublish, bool kJoin, typename C, typename X, typename S, typename F,
          typename O = NoScalars>
__device__ __forceinline__ bool exact_sum(const GridSync &gs, Episode &episode, ExactState &xs,
                                          SumWindow<NV> &win, int *part, C &&put, X &&expo,
                                          S &&side, F &&f, O &&overlap = O()) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (kPublish) ++episode.pub;
  bool first = true, have = true;
#pragma unroll
  for (int q = 0; q < NV; ++q) have = have && win.top[q] != kNoWindow;
#pragma unroll 1
  for (;;) {
    if (!have) {
      if (!window_by_partials(gs.slots, gs.count, gs.err, gs.nblocks, blockIdx.x - gs.base,
                              gs.cluster, ++episode.n, xs, win.top, NV, expo(0),
                              NV > 1 ? expo(1 % NV) : 0, NV > 2 ? expo(2 % NV) : 0, part))
        return false;
    }
    const unsigned int set = (episode.x++) & 1u;
#pragma unroll
    for (int q = 0; q < NV; ++q) put(q, win.top[q], xs.acc[set] + 8 * q);
    __syncthreads();
    if (warp == 0) {
      double t[NV];
      const int r = exact_words<NV>(gs.xw, gs.err, gs.nblocks, set, !have, win, xs, t);
      if (kJoin && first) join_warps01();
      if (lane == 0) {
        xs.flag = r;
        if (r == 1) {
          window_set<NV>(win, t);
          f(t);
        }
      }
    } else if (warp == 1) {
      if (lane == 0 && first) side();
      if (kJoin && first) join_warps01();
    } else if (kPublish && warp == 2 && first) {
      bool ok = true;  // (one block publishes by the __syncthreads)
      if (gs.nblocks > 1) {
        if (lane == 0) red_add_release(gs.count + 8, 1u);
        ok = wait_count<true>(gs.count + 8, gs.err, episode.pub * gs.nblocks);
      }
      if (lane == 0) xs.pub_ok = ok ? 1 : 0;
    } else if (warp >= 3 && first) {
      overlap();
    }
    __syncthreads();
    if (kPublish && !xs.pub_ok) return false;
    const int r = xs.flag;
    if (r != 2) return r == 1;
    first = false;
    have = false;
  }
}

// exact_sum of FP64 partials; buf: NV x blockDim doubles of shared memory.
template <int NV, bool kPublish, bool kJoin, typename S, typename F, typename O = NoScalars>
__device__ __forceinline__ bool grid_sum_x(const GridSync &gs, Episode &episode, ExactState &xs,
                                           SumWindow<NV> &win, const double (&v)[NV], double *buf,
                                           S &&side, F &&f, O &&overlap = O()) {
  return exact_sum<NV, kPublish, kJoin>(
      gs, episode, xs, win, reinterpret_cast<int *>(buf),
      [&](int q, int top, int *acc) { put_limbs(v[q], top, acc); },
      [&](int q) { return (__double2hiint(v[q]) >> 20) & 0x7ff; }, side, f, overlap);
}

// Streaming loads of read-only matrix data (never written by the kernel
// that reads them): non-coherent path, no L1 allocation.
__device__ __forceinline__ int ld_stream(const int *p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_stream(const double *p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int16_t ld_stream16(const int16_t *p) {
  short v;
  asm volatile("ld.global.nc.L1::no_allocate.s16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float *p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
// 16-byte and 8-byte streaming loads (p aligned to 16 / 8 bytes): one
// row's four FP32 weights, one row's four 16-bit column offsets.
__device__ __forceinline__ float4 ld_stream4(const float *p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_stream_u2(const int16_t *p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "l"(p));
  return v;
}
// The k-th signed 16-bit offset of four packed in (lo, hi) words.
__device__ __forceinline__ int off16(uint2 v, int k) {
  const unsigned int w = (k < 2) ? v.x : v.y;
  return (int)(int16_t)(uint16_t)((k & 1) ? (w >> 16) : (w & 0xffffu));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// y_row = (A x)_row for the lane's row of slice s, with x supplied by a
// functor (so callers can form x on the fly, e.g. p = z + beta*p).  Rows
// of width <= 4 (every cell of a triangle/quad mesh) issue all value and
// column loads before the gathers, so a warp has 8 independent streaming
// loads in flight per slice.
// Reference order: DIAG_FIRST  t = ad*x_i; t = t + a_k*x_k ...  (csrd)
//                  DIAG_LAST   t = a_1x_1 + ... + a_wx_w + ad*x_i (ellpack)
//                  DIAG_NONE   t = 0 + a_k*x_k ...                 (csr)
template <typename XF>
__device__ __forceinline__ double sell_row_f64(const SellView<double> &A, int s,
                                               int lane, int row, XF xf) {
  const int64_t base = A.sptr[s];
  int w = (int)((A.sptr[s + 1] - base) >> 5);
  FVC_CHK(w >= 0 && w <= A.n, A.chk, kChkSliceWidth, w = 0);
  const int *cp = A.col + base + lane;
  const double *vp = A.val + base + lane;
  double xd = 0.0;
  if (A.diag_mode != DIAG_NONE) xd = __dmul_rn(ld_stream(A.diag + row), xf(row));
  double t = (A.diag_mode == DIAG_FIRST) ? xd : 0.0;
  if (w <= 4) {
    int c[4];
    double a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = (k < w) ? ld_stream(cp + 32 * k) : 0;
      a[k] = (k < w) ? ld_stream(vp + 32 * k) : 0.0;
      FVC_CHK(k >= w || (unsigned)c[k] < (unsigned)A.n, A.chk, kChkColumn, c[k] = row);
    }
    if (A.diag_mode == DIAG_LAST) {
      // the reference's ELLPACK sums t1+t2+...+tw+t_diag left to right
      if (w > 0) t = __dmul_rn(a[0], xf(c[0]));
#pragma unroll
      for (int k = 1; k < 4; ++k)
        if (k < w) t = __dadd_rn(t, __dmul_rn(a[k], xf(c[k])));
      return __dadd_rn(t, xd);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < w) t = __dadd_rn(t, __dmul_rn(a[k], xf(c[k])));
    return t;
  }
  auto colk = [&](int k) {
    int c = ld_stream(cp + 32 * k);
    FVC_CHK((unsigned)c < (unsigned)A.n, A.chk, kChkColumn, c = row);
    return c;
  };
  if (A.diag_mode == DIAG_LAST) {
    t = __dmul_rn(ld_stream(vp), xf(colk(0)));
    for (int k = 1; k < w; ++k) t = __dadd_rn(t, __dmul_rn(ld_stream(vp + 32 * k), xf(colk(k))));
    return __dadd_rn(t, xd);
  }
  for (int k = 0; k < w; ++k) t = __dadd_rn(t, __dmul_rn(ld_stream(vp + 32 * k), xf(colk(k))));
  return t;
}

// The same row sum with fused multiply-adds (one FP64 instruction per
// term instead of two; GB300's FP64 pipe, ~1/64 of its FP32 rate, is the
// bottleneck of the FP64 solvers).  Terms are added in the same order.
// Wider rows go four entries at a time too: one at a time, the loads and the
// gather of each wait for the last (1M rows of eight: PCG 67 -> 50 us per
// iteration, BiCGSTAB 121 -> 92, transposed 183 -> 113, mixed BiCGSTAB 112 -> 75;
// 262k rows 20.7 -> 16.3, 40.5 -> 31.9, 45.3 -> 31.7, 36.5 -> 28.7).
// kUnrolled: the wider rows' loop as the compiler unrolls it (spmv_f64).
template <bool kUnrolled = false, typename XF>
__device__ __forceinline__ double sell_row_fma(const SellView<double> &A, int s, int lane,
                                               int row, XF xf) {
  const int64_t base = A.sptr[s];
  int w = (int)((A.sptr[s + 1] - base) >> 5);
  FVC_CHK(w >= 0 && w <= A.n, A.chk, kChkSliceWidth, w = 0);
  const int *cp = A.col + base + lane;
  const double *vp = A.val + base + lane;
  const bool has_diag = A.diag_mode != DIAG_NONE;
  const double dv = has_diag ? ld_stream(A.diag + row) : 0.0;
  const double xi = has_diag ? xf(row) : 0.0;
  double t = (A.diag_mode == DIAG_FIRST) ? dv * xi : 0.0;
  auto four = [&](int k0) {
    int c[4];
    double a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = k0 + k < w;
      c[k] = in ? ld_stream(cp + 32 * (k0 + k)) : 0;
      a[k] = in ? ld_stream(vp + 32 * (k0 + k)) : 0.0;
      FVC_CHK(!in || (unsigned)c[k] < (unsigned)A.n, A.chk, kChkColumn, c[k] = row);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k0 + k < w) t = fma(a[k], xf(c[k]), t);
  };
  if (w <= 4) {
    four(0);
  } else if (kUnrolled) {
    for (int k = 0; k < w; ++k) {
      int c = ld_stream(cp + 32 * k);
      FVC_CHK((unsigned)c < (unsigned)A.n, A.chk, kChkColumn, c = row);
      t = fma(ld_stream(vp + 32 * k), xf(c), t);
    }
  } else {
#pragma unroll 1
    for (int k0 = 0; k0 < w; k0 += 4) four(k0);
  }
  if (A.diag_mode == DIAG_LAST) t = fma(dv, xi, t);
  return t;
}

// One system of a batch: its slices, its solver (1 PCG, 2 BiCGSTAB), its
// stopping tolerance, inner tolerance (mixed precision) and warm-start
// rule, its synchronisation state (counter, partials, nblocks and first
// block) and its result slots.
struct BatchSys {
  int s0, s1;
  int code, init;
  double tol, inner_tol;
  GridSync gs;
  double *result;
  int *iresult;
  // per-system mask (may be null: always solve).  *run == 0: the system is
  // not solved in this launch -- the reference's test before a solve
  // (the right-hand side's norm below 1e-32) skipped it -- and x keeps its
  // rows' values
  const int32_t *run = nullptr;
};

// A masked system's blocks leave at once; its lead block reports status
// FVC_OK after 0 iterations.  Every block of the group reads the same flag.
__device__ __forceinline__ bool batch_masked(const BatchSys &d, bool lead) {
  if (d.run == nullptr || *d.run != 0) return false;
  if (lead && threadIdx.x == 0) {
    d.iresult[0] = 0;
    d.iresult[1] = FVC_OK;
    d.iresult[2] = 0;
  }
  return true;
}

// y_row = (A^T x)_row over the stored matrix of a symmetric pattern: the
// entry (row, col(slot)) of A^T is the stored value of the mirror slot
// (col(slot), row); the diagonal is A's.  Terms in slot order, with FMA.
template <typename XF>
__device__ __forceinline__ double sell_row_fma_t(const SellView<double> &A, int s, int lane,
                                                 int row, XF xf) {
  const int64_t base = A.sptr[s];
  int w = (int)((A.sptr[s + 1] - base) >> 5);
  FVC_CHK(w >= 0 && w <= A.n, A.chk, kChkSliceWidth, w = 0);
  const int *cp = A.col + base + lane;
  const int *mp = A.mirror + base + lane;
  const bool has_diag = A.diag_mode != DIAG_NONE;
  const double dv = has_diag ? ld_stream(A.diag + row) : 0.0;
  double t = has_diag ? dv * xf(row) : 0.0;
#ifdef FVC_CHECK
  const int64_t nslots = A.sptr[A.nslices];
#endif
  auto four = [&](int k0) {
    int c[4], m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = k0 + k < w;
      c[k] = in ? ld_stream(cp + 32 * (k0 + k)) : 0;
      m[k] = in ? ld_stream(mp + 32 * (k0 + k)) : 0;
      FVC_CHK(!in || (unsigned)c[k] < (unsigned)A.n, A.chk, kChkColumn, c[k] = row);
      FVC_CHK(!in || (m[k] >= 0 && m[k] < nslots), A.chk, kChkMirror, m[k] = (int)(base + lane));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k0 + k < w) t = fma(A.val[m[k]], xf(c[k]), t);
  };
  if (w <= 4) {
    four(0);
  } else {
#pragma unroll 1
    for (int k0 = 0; k0 < w; k0 += 4) four(k0);
  }
  return t;
}

// A x (kT false) or A^T x (kT true) for one row
template <bool kT, typename XF>
__device__ __forceinline__ double row_fma(const SellView<double> &A, int s, int lane, int row,
                                          XF xf) {
  if (kT) return sell_row_fma_t(A, s, lane, row, xf);
  return sell_row_fma(A, s, lane, row, xf);
}

// Host side: scratch for the grid synchronisation of a persistent launch.
// One buffer: counter (64 bytes) | error block (64) | result (16 doubles) |
// iresult (16 ints) | padding | the words of the exact sums | the reduction
// slots; one memset clears it.
constexpr size_t kXBytes = 2 * (size_t)kXWords * sizeof(unsigned long long);
constexpr size_t kSyncHead = 512 + kXBytes;
static_assert(64 + 64 + 16 * sizeof(double) + 16 * sizeof(int) <= 512, "sync header");
constexpr size_t kSyncBlocks = 1280;  // blocks the first allocation serves

inline size_t slot_bytes(size_t nblocks) { return 4 * kMaxNV * nblocks * sizeof(RedSlot); }

inline int32_t ensure_sync(Scratch &S, size_t nblocks) {
  if (S.nslot < nblocks) {
    const size_t cap = std::max(nblocks, kSyncBlocks);
    if (S.sync) cudaFree(S.sync);
    S.sync = nullptr;
    S.nslot = 0;
    char *buf = nullptr;
    if (cudaMalloc(&buf, kSyncHead + slot_bytes(cap)) != cudaSuccess ||
        cudaMemset(buf, 0, kSyncHead) != cudaSuccess)
      return FVC_ERR_CUDA;
    S.sync = reinterpret_cast<unsigned int *>(buf);
    S.err = reinterpret_cast<int *>(buf + 64);
    S.result = reinterpret_cast<double *>(buf + 128);
    S.iresult = reinterpret_cast<int *>(buf + 128 + 16 * sizeof(double));
    S.nslot = cap;
  }
  if (!S.trace) {
    if (cudaMalloc(&S.trace, 2 * kTraceMax * sizeof(double)) != cudaSuccess) return FVC_ERR_CUDA;
    if (cudaMalloc(&S.history, kHistoryMax * sizeof(float)) != cudaSuccess) return FVC_ERR_CUDA;
  }
  return FVC_OK;
}

inline GridSync make_sync(const Scratch &S, int nblocks) {
  GridSync g;
  g.count = S.sync;
  g.err = S.err;
  g.xw = reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(S.sync) + 512);
  g.slots = reinterpret_cast<RedSlot *>(reinterpret_cast<char *>(S.sync) + kSyncHead);
  g.nblocks = (unsigned int)nblocks;
  g.base = 0;
  return g;
}

// The word a failed device check records into (check builds): the second
// 32-byte sector of the launch's 64-byte error block, zeroed with it.  A
// separate word from the wait error, so that no wait gives up early (the
// staged kernels must see every bulk copy land); the launch runs to its end
// on the redirected indices and the host reads the word afterwards
// (check_word_status).
inline int *check_word(const Scratch &S) { return S.err ? S.err + 8 : nullptr; }
int32_t check_word_status(const Scratch &S, cudaStream_t stream);

// The counter, error block, results and the slots of nblocks blocks start
// at zero (nblocks 0: a launch that reduces through its cluster).
inline void reset_sync(Scratch &S, cudaStream_t stream, size_t nblocks) {
  cudaMemsetAsync(S.sync, 0, kSyncHead + slot_bytes(nblocks), stream);
}

}  // namespace fvc
