// fvc_cluster.cu -- Jacobi-PCG (src/Iterativos.f:29-106) of a small system
// on one thread-block cluster, resident in its registers and shared memory.
//
// A system of a few thousand rows (the SIMPLE p' system of a 64 x 64 cavity
// has 4096) leaves a grid-wide persistent kernel latency-bound: every
// iteration waits twice for all blocks through L2.  Here the rows are split
// over the CTAs of one cluster (up to 16 SMs), one row per thread: its matrix
// row, x, r, p, q and 1/m stay in registers, p also in shared memory, where the
// SpMV of the other CTAs reads it (DSMEM).  Sums are exact integer sums
// (fvc_device.cuh), the CTAs' limbs exchanged by one cluster barrier: every
// CTA posts its limbs in its own shared memory, and after the barrier every
// CTA adds all of them itself (identical totals in every CTA, so every CTA
// takes the same branch).  Per iteration: form p, barrier, SpMV + p.q, sum,
// update + r.z, sum -- three cluster barriers and no global-memory traffic;
// x += alpha p runs between the arrival and the wait of the last one.
//
// What bounds it: chains of dependent FP64 instructions (64 clocks each; two
// warps of an SM sub-partition share a pipe that takes one per 76 clocks) and
// the barriers (420 clocks, and 230 for the DSMEM read after each).  Of the
// 6,900 clocks of an iteration at 2304 rows each sum takes some 1,800, the SpMV
// 1,100, the scalars between 300 (alpha) and 400 (beta, the stopping test).
// Per iteration, against rows in shared memory and sums in FP64: 256 rows 3.3
// us, 1024 rows 3.3, 2304 rows 3.5 against 6.4, 4096 rows 3.6 against 6.7, 8100
// rows 4.4 against 8.4.
//
// There is no spin-wait: the only waits are hardware cluster barriers, which
// every CTA reaches the same number of times (the loop exit depends only on
// the identical totals and maxit), and a last barrier keeps every CTA's
// shared memory alive until the others have finished reading it.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "fvc_device.cuh"
#include "fvc_internal.h"

namespace cg = cooperative_groups;

namespace fvc {
namespace {

constexpr int kClMax = 16;        // CTAs per cluster (non-portable above 8)
constexpr int kClMaxRows = 512;   // rows per CTA: one per thread
// Largest system run on a cluster: per iteration against the grid-wide kernel
// (128-thread blocks), 4096 rows 3.6 and 5.6 us, 8100 rows 4.4 and 6.1.
constexpr int kClMaxN = 8192;

struct ClArgs {
  SellView<double> A;
  const double *minv, *b;
  double *x;
  int R;            // rows per CTA, a multiple of 32
  double tol;
  int maxit, init, stop_rule;
  double *result;   // [0] energy [1] conv [2] final_crit [3] |b-Ax|^2 [4] |b|^2
  int *iresult;     // [0] iterations [1] status
};

// shared-memory layout of one CTA (R rows, S slots): p and x, and the slots
// beyond the fourth of a row are read from the staged copy
struct ClLayout {
  int R, S;
  __host__ __device__ size_t bytes() const {
    return (size_t)2 * R * sizeof(double) + (size_t)S * (sizeof(double) + sizeof(int)) +
           (size_t)(R / 32 + 1) * sizeof(int);
  }
};

extern __shared__ __align__(16) unsigned char cl_smem[];

// sqrt_bound's bound with room for the roundings between t[0] and beta d
__device__ __forceinline__ long long far_bound(long long bound) {
  return bound >= 0x7ff0000000000000ll ? 0x7fffffffffffffffll : bound + 16;
}
__device__ __forceinline__ bool middling(double v) {
  const int e = (__double2hiint(v) >> 20) & 0x7ff;
  return e > 1023 - 500 && e < 1023 + 500;
}

// The cluster's state of its sums (shared memory of each CTA): ExactState
// without the words, and the two sets of posted limbs.
struct ClSum {
  ExactState xs;
  long long post[2][32];
  alignas(8) int part[6 * 32];  // ordered: 3 x 32 doubles
};

// The same sum added in FP64 in a fixed order (Scratch::ordered): a shuffle
// tree per warp, one over the warps, one over the CTAs.
template <int NV, typename O, typename S, typename F>
__device__ __forceinline__ void cluster_sum_ordered(cg::cluster_group &cl, unsigned int &ep,
                                                    ClSum &cs, const double (&v)[NV], O &&overlap,
                                                    S &&side, F &&f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned int set = ep++ & 1u;
  double *part = reinterpret_cast<double *>(cs.part);
  double *post = reinterpret_cast<double *>(cs.post[set]);
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const double t = warp_sum(v[q]);
    if (lane == 0) part[q * 32 + warp] = t;
  }
  __syncthreads();
  if (warp == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const double t = warp_sum(lane < nw ? part[q * 32 + lane] : 0.0);
      if (lane == 0) post[q] = t;
    }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  overlap();
  if (threadIdx.x == 32) side();
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (warp == 0) {
    const int nb = (int)cl.num_blocks();
    double t[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q)
      t[q] = warp_sum(lane < nb ? *cl.map_shared_rank(post + q, lane) : 0.0);
    if (lane == 0) f(t);
  }
  __syncthreads();
}

// The exact sum (see exact_sum) over a cluster.  overlap() runs in every
// thread, side() in thread 32, between the arrival at the cluster barrier and
// its wait; f(totals) in thread 0.
template <bool kOrdered, int NV, typename O, typename S, typename F>
__device__ __forceinline__ void cluster_sum(cg::cluster_group &cl, unsigned int &ep, ClSum &cs,
                                            SumWindow<NV> &win, const double (&v)[NV],
                                            O &&overlap, S &&side, F &&f) {
  if (kOrdered) return cluster_sum_ordered<NV>(cl, ep, cs, v, overlap, side, f);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nb = (int)cl.num_blocks();
  ExactState &xs = cs.xs;
  bool first = true, have = true;
#pragma unroll
  for (int q = 0; q < NV; ++q) have = have && win.top[q] != kNoWindow;
#pragma unroll 1
  for (;;) {
    if (!have) {  // the window from the largest partial of the cluster
      const unsigned int set = ep++ & 1u;
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const int m = __reduce_max_sync(0xffffffffu, (__double2hiint(v[q]) >> 20) & 0x7ff);
        if (lane == 0) cs.part[q * 32 + warp] = m;
      }
      __syncthreads();
      if (warp == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          const int m = __reduce_max_sync(0xffffffffu, lane < nw ? cs.part[q * 32 + lane] : 0);
          if (lane == 0) cs.post[set][q] = m;
        }
      cl.sync();
      if (warp == 0) {
        bool nan = false;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          const int m = __reduce_max_sync(
              0xffffffffu, lane < nb ? (int)*cl.map_shared_rank(&cs.post[set][q], lane) : 0);
          nan = nan || m == 0x7ff;
          if (lane == 0) win.top[q] = top_of_partials(m);
        }
        if (lane == 0) xs.nan = nan ? 1 : 0;
      }
      __syncthreads();
    }
    const unsigned int set = ep++ & 1u;
#pragma unroll
    for (int q = 0; q < NV; ++q) put_limbs(v[q], win.top[q], xs.acc[set] + 8 * q);
    __syncthreads();
    if (warp == 0) cs.post[set][lane] = block_limbs(xs.acc[set]);
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (first) {
      overlap();
      if (threadIdx.x == 32) side();
      __syncwarp();
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (warp == 0) {
      // every lane reads kClMax / kG CTAs' words, the lanes add theirs
      constexpr int kG = NV == 1 ? 4 : NV == 2 ? 2 : 1, kW = 32 / kG;
      long long d[kClMax / kG], s = 0;
#pragma unroll
      for (int i = 0; i < kClMax / kG; ++i) {
        const int c = i * kG + lane / kW;
        d[i] = (c < nb) ? *cl.map_shared_rank(&cs.post[set][lane % kW], c) : 0;
      }
#pragma unroll
      for (int i = 0; i < kClMax / kG; ++i) s += d[i];
#pragma unroll
      for (int o = kW; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const long long L = (long long)((unsigned long long)s << 22) >> 22;
      double t[NV];
      const int r = limb_totals<NV>(L, ((s - L) >> 42) != 0, true, !have, win, xs, t);
      if (lane == 0) {
        xs.flag = r;
        if (r == 1) {
          window_set<NV>(win, t);
          f(t);
        }
      }
      __syncwarp();
    }
    __syncthreads();
    if (xs.flag == 1) return;
    first = false;
    have = false;
  }
}

template <bool kOrdered>
__global__ void __launch_bounds__(kClMaxRows, 1) pcg_cluster(ClArgs a) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClSum cs;
  __shared__ SumWindow<1> wpq, wrz;
  __shared__ SumWindow<2> wrr;
  __shared__ SumWindow<3> w3;
  __shared__ struct {
    double d, alpha, beta, conv, crit2;
    Divisor dv;
    long long bound, far;  // of the stopping test
    int stop;
  } sh;
  const int rank = (int)cl.block_rank(), nb = (int)cl.num_blocks();
  const int R = a.R, n = a.A.n;
  const int r0 = rank * R;
  const int rows = max(0, min(R, n - r0));
  const int ns = (rows + 31) / 32, s0 = r0 / 32;
  const int64_t sbase = a.A.sptr[s0];
  const int S = (int)(a.A.sptr[s0 + ns] - sbase);
  double *p = reinterpret_cast<double *>(cl_smem);  // read by the other CTAs
  double *xv = p + R;                               // so is x, before and after the loop
  double *val = xv + R;
  int *col = reinterpret_cast<int *>(val + S);  // (owner << 16) | local row
  int *sp = col + S;                            // slot offset of each local slice
  const bool has_diag = a.A.diag_mode != DIAG_NONE;
  exact_init(cs.xs);
  if (threadIdx.x == 0) wpq.top[0] = wrz.top[0] = wrr.top[0] = w3.top[0] = kNoWindow;
#ifdef FVC_CHECK
  // check builds: columns outside [0, n) (whose owner CTA would not be in
  // the cluster) are counted here, redirected to this CTA's first row, and
  // end the solve uniformly after the first reduction
  __shared__ int s_bad;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
#endif
  // load the rows' slices (columns re-coded as owner CTA and local row)
  for (int i = threadIdx.x; i <= ns; i += blockDim.x) sp[i] = (int)(a.A.sptr[s0 + i] - sbase);
  for (int k = threadIdx.x; k < S; k += blockDim.x) {
    int c = a.A.col[sbase + k];
    FVC_CHK((unsigned)c < (unsigned)n, &s_bad, kChkCluster, c = r0);
    const int owner = c / R;
    col[k] = (owner << 16) | (c - owner * R);
    val[k] = a.A.val[sbase + k];
  }
  // this thread's row (blockDim >= R)
  const int i = threadIdx.x;
  const bool own = i < rows;
  const double mi = own ? a.minv[r0 + i] : 0.0;
  const double dg = (own && has_diag) ? a.A.diag[r0 + i] : 0.0;
  const double bi = own ? a.b[r0 + i] : 0.0;
  double x = (own && !a.init) ? a.x[r0 + i] : 0.0;
  if (i < R) {
    p[i] = 0.0;
    xv[i] = x;
  }
  cl.sync();  // every CTA's x in place
  // its first four slots in registers: values, and where the neighbours' p are
  int w = 0, base = 0;
  double v4[4] = {0.0, 0.0, 0.0, 0.0};
  const double *nb4[4] = {p, p, p, p};
  if (own) {
    base = sp[i >> 5] + (i & 31);
    w = (sp[(i >> 5) + 1] - sp[i >> 5]) >> 5;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < w) {
        const int c = col[base + 32 * k], o = c >> 16, l = c & 0xffff;
        v4[k] = val[base + 32 * k];
        nb4[k] = (o == rank) ? p + l : cl.map_shared_rank(p, o) + l;
      }
  }
  const ptrdiff_t dx = xv - p;  // x beside p in every CTA
  // (A u)_i in the reference's diagonal order; off: where u lies from p
  auto spmv_row = [&](double ui, ptrdiff_t off) -> double {
    double u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = (k < w) ? nb4[k][off] : 0.0;
    double t = (a.A.diag_mode == DIAG_FIRST) ? dg * ui : 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < w) t = fma(v4[k], u[k], t);
#pragma unroll 1
    for (int k = 4; k < w; ++k) {
      const int c = col[base + 32 * k], o = c >> 16, l = c & 0xffff;
      const double *q = (o == rank) ? p : cl.map_shared_rank(p, o);
      t = fma(val[base + 32 * k], q[l + off], t);
    }
    if (a.A.diag_mode == DIAG_LAST) t = fma(dg, ui, t);
    return t;
  };

  unsigned int ep = 0;
  const bool rule0 = a.stop_rule == 0;
  auto none = [] {};
  // r = b - A x ; z = r/m ; p = z ; d = r.z
  double r = own ? bi - (a.init ? 0.0 : spmv_row(x, dx)) : 0.0;
  double z = r * mi;
#ifdef FVC_CHECK
  double acc[3] = {r * z, bi * bi, (threadIdx.x == 0 && s_bad != 0) ? 1.0 : 0.0};
  __syncthreads();
  cluster_sum<kOrdered, 3>(cl, ep, cs, w3, acc, none, none, [&](const double *t) {
    sh.stop = (t[2] > 0.0) ? 3 : 0;
#else
  double acc[2] = {r * z, bi * bi};
  cluster_sum<kOrdered, 2>(cl, ep, cs, wrr, acc, none, none, [&](const double *t) {
    sh.stop = 0;
#endif
    sh.d = t[0];
    sh.conv = a.tol * root(rule0 ? fabs(t[0]) : t[1]);
    sh.bound = sqrt_bound(sh.conv);
    sh.far = far_bound(sh.bound);
    sh.crit2 = 0.0;
    wrz.top[0] = window_top(t[0]);
    wrr.top[1] = kNoWindow;
  });
  int j, status = FVC_OK;
  double beta = 0.0, pi = 0.0;
  const int jmax = (sh.stop == 3) ? 0 : a.maxit;  // 3: a failed check (check builds)
  if (sh.stop == 3) status = FVC_ERR_ARG;
#pragma unroll 1
  for (j = 1; j <= jmax; ++j) {
    // p = z + beta p on the own rows (the first: p = z), then visible to the cluster
    pi = fma(beta, pi, z);
    if (i < R) p[i] = pi;
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (threadIdx.x == 0 && j > 1) sh.d = sh.beta * sh.d;  // read after the next __syncthreads
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    const double qi = own ? spmv_row(pi, 0) : 0.0;
    const double pq[1] = {pi * qi};
    cluster_sum<kOrdered, 1>(cl, ep, cs, wpq, pq, none, [&] { sh.dv.set(sh.d); },
                   [&](const double *t) {
                     sh.alpha = kOrdered ? divide(sh.d, t[0]) : quick_quotient(sh.d, t[0]);
                   });
    const double alpha = sh.alpha;
    r = fma(-alpha, qi, r);
    z = r * mi;
    // beta = r.z / d ; the next d = beta d, formed while the next barrier is
    // waited for; the reference's stopping test.  Far from its bound the test
    // needs neither d nor a root: beta d is t[0] to two roundings (exponents
    // within +-500 of 1)
    auto step = [&](const double *t) {
      const double b = quotient(t[0], sh.dv);
      sh.beta = b;
      const double c = rule0 ? t[0] : t[rule0 ? 0 : 1];
      if (middling(t[0]) && middling(b) && __double_as_longlong(c) > sh.far && !is_nan_bits(c)) {
        sh.stop = 0;
        if (!rule0) sh.crit2 = c;
        return;
      }
      const double d = b * sh.d;
      const double crit2 = rule0 ? fabs(d) : c;
      sh.crit2 = crit2;
      sh.stop = (is_nan_bits(crit2) || not_finite_bits(d)) ? 2
                : sqrt_below(crit2, sh.conv, sh.bound)     ? 1
                                                           : 0;
    };
    auto update_x = [&] { x = fma(alpha, pi, x); };
    if (rule0) {
      const double rz[1] = {r * z};
      cluster_sum<kOrdered, 1>(cl, ep, cs, wrz, rz, update_x, none, step);
    } else {
      const double rr[2] = {r * z, r * r};
      cluster_sum<kOrdered, 2>(cl, ep, cs, wrr, rr, update_x, none, step);
    }
    if (sh.stop == 2) {
      status = FVC_ERR_NAN;
      break;
    }
    if (sh.stop == 1) break;
    beta = sh.beta;
  }
  if (j > a.maxit && status == FVC_OK) {
    j = a.maxit;
    status = FVC_ERR_NOCONV;
    if (rule0 && j > 0 && threadIdx.x == 0) sh.crit2 = fabs(sh.beta * sh.d);
  }
  if (status == FVC_ERR_ARG) j = 0;
  // x.Ax, |b - Ax|^2, |b|^2 (x complete in every CTA after the barrier)
  if (i < R) xv[i] = x;
  if (threadIdx.x == 0) w3.top[0] = kNoWindow;
  cl.sync();
  double e3[3] = {0.0, 0.0, 0.0};
  if (own) {
    const double ax = spmv_row(x, dx), rr = bi - ax;
    e3[0] = x * ax;
    e3[1] = rr * rr;
    e3[2] = bi * bi;
    a.x[r0 + i] = x;
  }
  cluster_sum<kOrdered, 3>(cl, ep, cs, w3, e3, none, none, [&](const double *t) {
    if (rank == 0) {
      a.result[0] = t[0];
      a.result[1] = sh.conv;
      a.result[2] = root(sh.crit2);
      a.result[3] = t[1];
      a.result[4] = t[2];
      a.iresult[0] = j;
      a.iresult[1] = status;
      a.iresult[2] = 0;
    }
  });
  cl.sync();  // no CTA leaves while another may still read its shared memory
}

// The cluster layout of an n-row system: CTAs, rows per CTA (a multiple of
// 32, at most kClMaxRows, over at most kClMax CTAs).  False when the system
// does not fit one cluster.
// One warp of rows per SM sub-partition while 16 CTAs hold them (an FP64
// instruction of a warp takes its sub-partition's pipe for 76 clocks), two for
// ordered sums, whose order the split is part of.
bool cluster_shape(int n, bool ordered, int &nb, int &R) {
  if (n <= 0 || n > kClMaxN) return false;
  const int per = ordered ? 256 : 128;
  nb = std::min(kClMax, std::max(1, (n + per - 1) / per));
  R = ((n + nb - 1) / nb + 31) / 32 * 32;
  if (R > kClMaxRows) return false;
  nb = (n + R - 1) / R;
  return true;
}

}  // namespace

// Largest number of stored slots of one CTA's rows under the cluster
// layout, from the host copy of the slice pointers; -1 when the system does
// not fit one cluster.
int cluster_slots_max(int n, int nslices, const int64_t *sptr) {
  int smax = sptr ? 0 : -1;
  for (const bool ordered : {false, true}) {  // the larger serves both
    int nb = 0, R = 0;
    if (!sptr || !cluster_shape(n, ordered, nb, R)) return -1;
    for (int c = 0; c < nb; ++c) {
      const int s0 = c * R / 32, s1 = std::min(nslices, (c + 1) * R / 32);
      smax = std::max(smax, (int)(sptr[s1] - sptr[s0]));
    }
  }
  return smax;
}

// Enqueues the cluster PCG when the system fits one cluster and returns
// without waiting; FVC_ERR_UNSUPPORTED (and nothing enqueued) when it does
// not, so the caller falls back to the grid-wide kernel.  launch = false
// only checks the fit and prepares the scratch.
int32_t enqueue_pcg_cluster(const DeviceMatrix &A, Scratch &S, const double *b, double *x,
                            double tol, int maxit, int init, const fvc_opts &o,
                            cudaStream_t stream, bool launch) {
  const int n = A.n;
  if (n <= 0 || A.diag_mode == DIAG_NONE || !A.jinv) return FVC_ERR_UNSUPPORTED;
  int nb = 0, R = 0;
  if (!cluster_shape(n, S.ordered, nb, R)) return FVC_ERR_UNSUPPORTED;
  int smax = A.cl_smax;
  if (smax < 0) {  // a matrix loaded without the host-side count
    std::vector<int64_t> sptr((size_t)A.nslices + 1);
    if (cudaMemcpyAsync(sptr.data(), A.sptr, sizeof(int64_t) * sptr.size(),
                        cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
      return FVC_ERR_CUDA;
    smax = cluster_slots_max(n, A.nslices, sptr.data());
  }
  const ClLayout L{R, smax};
  const size_t smem = L.bytes();
  if (smem > 200 * 1024) return FVC_ERR_UNSUPPORTED;
  auto *kern = S.ordered ? pcg_cluster<true> : pcg_cluster<false>;
  static bool attrs_set = false;
  if (!attrs_set) {
    for (auto *k : {pcg_cluster<false>, pcg_cluster<true>}) {
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    attrs_set = true;
  }
  const int threads = std::min(1024, std::max(128, (R + 127) / 128 * 128));
  if (ensure_sync(S, 1) != FVC_OK) return FVC_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nb);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)nb;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess ||
      clusters < 1) {
    cudaGetLastError();
    return FVC_ERR_UNSUPPORTED;
  }
  if (!launch) return FVC_OK;
  reset_sync(S, stream, 0);
  ClArgs a{};
  a.A = SellView<double>{A.n, A.nslices, A.sptr, A.col, A.val, A.diag, A.diag_mode};
  a.minv = A.jinv;
  a.b = b;
  a.x = x;
  a.R = R;
  a.tol = tol;
  a.maxit = maxit;
  a.init = init;
  a.stop_rule = o.stop_rule;
  a.result = S.result;
  a.iresult = S.iresult;
  const cudaError_t ce = cudaLaunchKernelEx(&cfg, kern, a);
  count_launch();
  if (ce != cudaSuccess) {
    fprintf(stderr, "fvcgpu: cluster PCG launch failed: %s\n", cudaGetErrorString(ce));
    cudaGetLastError();
    return FVC_ERR_CUDA;
  }
  return FVC_OK;
}

// Runs the cluster PCG synchronously (FVC_ERR_UNSUPPORTED when the system
// does not fit one cluster).
int32_t run_pcg_cluster(const DeviceMatrix &A, Scratch &S, const double *b, double *x,
                        double tol, int maxit, int init, const fvc_opts &o, cudaStream_t stream,
                        fvc_stats *st) {
  int32_t rc = enqueue_pcg_cluster(A, S, b, x, tol, maxit, init, o, stream, false);
  if (rc != FVC_OK) return rc;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, stream);
  rc = enqueue_pcg_cluster(A, S, b, x, tol, maxit, init, o, stream, true);
  cudaEventRecord(e1, stream);
  if (rc != FVC_OK) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
  }
  double res[16];
  int ires[16];
  cudaMemcpyAsync(res, S.result, sizeof(res), cudaMemcpyDeviceToHost, stream);
  cudaMemcpyAsync(ires, S.iresult, sizeof(ires), cudaMemcpyDeviceToHost, stream);
  const cudaError_t ce = cudaStreamSynchronize(stream);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ce != cudaSuccess) {
    fprintf(stderr, "fvcgpu: cluster PCG failed: %s\n", cudaGetErrorString(ce));
    return FVC_ERR_CUDA;
  }
#ifdef FVC_CHECK
  if (ires[1] == FVC_ERR_ARG)
    fprintf(stderr, "fvcgpu: device check failed: cluster PCG column outside [0, n) (code %d); "
                    "the solve's result is void\n", (int)kChkCluster);
#endif
  if (st) {
    st->status = ires[1];
    st->iterations = ires[0];
    st->inner_iterations = 0;
    st->refinements = 0;
    st->energy = res[0];
    st->conv = res[1];
    st->final_crit = res[2];
    st->rel_residual = (res[4] > 0) ? std::sqrt(res[3] / res[4]) : std::sqrt(res[3]);
    st->solve_ms = ms;
  }
  return ires[1];
}

}  // namespace fvc
