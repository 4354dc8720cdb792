// gjx_kernels.cu -- the kernels of a single decomposition: one launch per outer
// step (clusters of CTAs per block pair, or two pairs per CTA), one per sweep,
// the reference's alternative builds; D, V and the tensor maps.
#include <cudaTypedefs.h>

#include "gjx_pair.cuh"

namespace gjx {

// one launch per outer step: block pair blockIdx.x / NSPLIT, cluster rank
// blockIdx.x % NSPLIT
template <bool SORT, bool ACCV, unsigned NSPLIT>
__global__ void __launch_bounds__(kThreads, 1) l1_step_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  pdl_launch();
  const unsigned rank = (NSPLIT > 1u) ? (blockIdx.x % NSPLIT) : 0u;
  pair_step<SORT, ACCV, NSPLIT, UpdBuffers<NSPLIT>::value>(P, P.step, blockIdx.x / NSPLIT, rank, sm);
}

// one launch per outer step, two block pairs per CTA (a step with more pairs
// than SMs: one wave instead of two, and the two pairs' serial phases
// overlap): CTA c takes pairs 2c and 2c + 1 through pair_step2, or the last
// pair alone through pair_step
template <bool SORT, bool ACCV>
__global__ void __launch_bounds__(kThreads, 1) l1_step2_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  pdl_launch();
  const unsigned a = 2u * blockIdx.x;
  if (a + 1u < P.pairs)
    pair_step2<SORT, ACCV>(P, P.step, a, P, P.step, a + 1u, sm);
  else
    pair_step<SORT, ACCV, 1u>(P, P.step, a, 0u, sm);
}

// one launch per outer step, one block pair per CTA of 4 warps, two CTAs per
// SM, up to its transform (P.vt): a step with more pairs than SMs
template <bool SORT>
__global__ void __launch_bounds__(kNThreads, 2) l1_stepn_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  pdl_launch();
  pair_step_n<SORT, false>(P, P.step, blockIdx.x, sm);
}

// ---------------------------------------------------------------------------
// The update of a step by itself: [G_i G_j] <- [G_i G_j] V_loc, and V likewise,
// for all block pairs (P.vt, P.vflag).  The 256-row stages of all pairs, in
// order, are dealt out evenly to one CTA per SM; a CTA takes a contiguous run,
// so its transform changes rarely (two buffers, the next pair's loaded with
// its first stage).  Stages as in pair_step with three buffers, the warps not
// waiting for one another.
// ---------------------------------------------------------------------------
constexpr unsigned kUOffVT = 3u * kUpdStage;
constexpr unsigned kUOffBar = kUOffVT + 2u * kTransform; // [0..2] stages, [3..4] transforms, [5..7] stages done
constexpr unsigned kUSmemDoubles = kUOffBar + 8u;
static_assert(kUSmemDoubles * sizeof(double) <= 227u * 1024u, "three stages and two transforms must fit");

template <bool ACCV>
__global__ void __launch_bounds__(kThreads, 1) l1_update_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kUOffBar);
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const unsigned nG = (P.nrow + kUpdRows - 1u) / kUpdRows;
  const unsigned nst = nG + (ACCV ? (P.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  const unsigned total = P.pairs * nst, per = total / gridDim.x, extra = total % gridDim.x;
  const unsigned first = blockIdx.x * per + min(blockIdx.x, extra);
  const unsigned end = first + per + (blockIdx.x < extra ? 1u : 0u);
  // the first stage from i on whose pair changes
  const auto live = [&](unsigned i) {
    while (i < end && !P.vflag[i / nst])
      i = (i / nst + 1u) * nst;
    return min(i, end);
  };
  const auto stage_at = [&](const unsigned i, const CUtensorMap *&tm, int &piece, int &ci, int &cj) {
    const unsigned pair = i / nst, k = i - pair * nst;
    const size_t pidx = ((size_t)P.step * P.pairs + pair) * 2u;
    tm = (k < nG) ? &P.tmG : &P.tmV;
    piece = (int)((((k < nG) ? k : (k - nG)) * kUpdRows) >> 5);
    ci = (int)(P.strat1[pidx] * kNColB);
    cj = (int)(P.strat1[pidx + 1u] * kNColB);
  };
  const auto load = [&](const unsigned i, const unsigned n) { // one thread: stage i as the n-th, 2 tensor copies
    const CUtensorMap *tm;
    int piece, ci, cj;
    stage_at(i, tm, piece, ci, cj);
    double *const st = sm + (n % 3u) * kUpdStage;
    mbar_arrive_expect_tx(&bars[n % 3u], 2u * kUpdBoxBytes);
    tma_load_3d(st, tm, 0, piece, ci, &bars[n % 3u]);
    tma_load_3d(st + 16u * kUpdColLd, tm, 0, piece, cj, &bars[n % 3u]);
  };
  const auto load_vt = [&](const unsigned pair, const unsigned m) { // one thread: the CTA's m-th transform
    mbar_arrive_expect_tx(&bars[3u + (m & 1u)], kTransform * 8u);
    bulk_g2s(sm + kUOffVT + (m & 1u) * kTransform, P.vt + (size_t)pair * kTransform, kTransform * 8u,
             &bars[3u + (m & 1u)]);
  };
  const auto store = [&](const unsigned i, const unsigned n) { // one thread: stage i, the n-th, back
    const CUtensorMap *tm;
    int piece, ci, cj;
    stage_at(i, tm, piece, ci, cj);
    const double *const st = sm + (n % 3u) * kUpdStage;
    tma_store_3d(tm, st, 0, piece, ci);
    tma_store_3d(tm, st + 16u * kUpdColLd, 0, piece, cj);
    bulk_commit();
  };
  const auto wait_done = [&](const unsigned n) { return mbar_wait_bounded(&bars[5u + n % 3u], (n / 3u) & 1u, kWaitLimit); };
  pdl_launch();
  pdl_wait(); // the transforms, G and V are the launch before's
  unsigned i = live(first);
  if (i >= end)
    return;
  __shared__ unsigned s_stop;
  volatile unsigned *const stop = &s_stop; // a wait gave up: all warps leave
  if (tid == 0u) {
    for (unsigned b = 0u; b < 8u; ++b)
      mbar_init(&bars[b], (b < 5u) ? 1u : kThreads / 32u);
    mbar_fence_init();
    *stop = 0u;
    load_vt(i / nst, 0u);
    load(i, 0u);
  }
  __syncthreads();
  const unsigned sub = lane & 7u, cg8 = lane >> 3;
  unsigned n = 0u, m = 0u, last = i, stages = 1u, transforms = 1u; // (the last two: thread 0's loads)
  int fail = 0;
  for (bool fresh = true; i < end; ++n) { // the n-th stage, with the m-th transform
    const unsigned j = live(i + 1u);
    const bool turn = j < end && j / nst != i / nst;
    if (tid == 0u) {
      if (n > 0u) {
        if (wait_done(n - 1u))
          store(last, n - 1u);
        else
          fail = 1;
      }
      if (j < end && !fail) {
        bulk_wait_read_but1(); // the store of the stage before the last has read its buffer out
        load(j, n + 1u);
        ++stages;
        if (turn) { // every warp is past the transform before the last
          load_vt(j / nst, m + 1u);
          ++transforms;
        }
      }
    }
    bool ok = !fail && !*stop;
    ok = ok && (!fresh || mbar_wait_bounded(&bars[3u + (m & 1u)], (m >> 1) & 1u, kWaitLimit));
    ok = ok && mbar_wait_bounded(&bars[n % 3u], (n / 3u) & 1u, kWaitLimit);
    fail = !__all_sync(0xffffffffu, ok);
    if (fail) {
      *stop = 1u;
      break;
    }
    double *const st = sm + (n % 3u) * kUpdStage;
    double acc[4][8];
    update_stage(st, sm + kUOffVT + (m & 1u) * kTransform, warp, sub, cg8, acc);
    __syncwarp();
    update_put(st, acc, warp, sub, cg8);
    fence_async_shared();
    __syncwarp();
    if (lane == 0u)
      mbar_arrive(&bars[5u + n % 3u]);
    fresh = turn;
    m += turn ? 1u : 0u;
    last = i;
    i = j;
  }
  if (tid == 0u && !fail) {
    if (wait_done(n - 1u))
      store(last, n - 1u);
    else
      fail = 1;
  }
  fail = __syncthreads_or(fail);
  if (tid == 0u) {
    if (fail) { // the copies in flight land (bounded); report
      for (unsigned q = (stages > 2u) ? stages - 2u : 0u; q < stages; ++q)
        (void)mbar_wait_bounded(&bars[q % 3u], (q / 3u) & 1u, kWaitLimit / 8);
      for (unsigned q = (transforms > 2u) ? transforms - 2u : 0u; q < transforms; ++q)
        (void)mbar_wait_bounded(&bars[3u + (q & 1u)], (q >> 1) & 1u, kWaitLimit / 8);
      atomicOr(P.err, kErrWaitTimeout);
    }
    bulk_wait_all();
  }
}

// the reference's alternative builds (P.variant: 1 -DUSE_QR, 2 -DUSE_DRMAC):
// one CTA per block pair, the QR factor in place of the Gram and Cholesky
template <bool SORT, bool ACCV, unsigned FAC>
__global__ void __launch_bounds__(kThreads, 1) l1_var_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  pair_step<SORT, ACCV, 1u, 2u, FAC>(P, P.step, blockIdx.x, 0u, sm);
}

// ---------------------------------------------------------------------------
// One launch for a whole sweep.  Cluster c takes block pair c of every outer
// step in turn.  A block is rewritten by exactly one pair per step, so pair
// (i, j) of step s may start once both blocks have been written by all CTAs
// of their step s-1 pairs: P.ver counts those CTAs (NSPLIT per step).
// Thread 0 of each CTA waits for the counts (bounded); the CTAs of a cluster
// agree through distributed shared memory and a cluster barrier, so they
// leave together on an error (pair_step has one cluster barrier on every
// path).  Writers fence their stores before counting; readers acquire the
// counts and fence the async proxy before their tile copies.  All clusters
// are resident at once (cooperative launch, checked on the host).
// ---------------------------------------------------------------------------
template <bool SORT, bool ACCV, unsigned NSPLIT>
__global__ void __launch_bounds__(kThreads, 1) l1_sweep_kernel(const __grid_constant__ StepParams P)
{
  extern __shared__ __align__(128) double sm[];
  __shared__ unsigned agree[NSPLIT]; // [r]: CTA r of the cluster may proceed
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kOffBar);
  const unsigned rank = (NSPLIT > 1u) ? (blockIdx.x % NSPLIT) : 0u;
  const unsigned pair = blockIdx.x / NSPLIT;
  if (NSPLIT > 1u) { // agree[] below is the cluster's first remote store
    cluster_started();
    cluster_wait_started();
  }
  for (unsigned step = 0u; step < P.steps1; ++step) {
    const size_t pidx = ((size_t)step * P.pairs + pair) * 2u;
    const unsigned iB = P.strat1[pidx + 0u], jB = P.strat1[pidx + 1u];
    if (threadIdx.x == 0u) {
      const unsigned need = NSPLIT * step;
      unsigned ok = (*(volatile int *)P.err == 0) ? 1u : 0u;
      const long long t0 = clock64();
      while (ok && (ld_acquire(P.ver + iB) < need || ld_acquire(P.ver + jB) < need)) {
        if (*(volatile int *)P.err)
          ok = 0u;
        else if (clock64() - t0 > kWaitLimit) {
          atomicOr(P.err, kErrWaitTimeout);
          ok = 0u;
        }
        else
          __nanosleep(64);
      }
      for (unsigned q = 0u; q < NSPLIT; ++q)
        cg::this_cluster().map_shared_rank(agree, q)[rank] = ok;
    }
    if (NSPLIT > 1u)
      cg::this_cluster().sync();
    else
      __syncthreads();
    unsigned all = 1u;
    for (unsigned q = 0u; q < NSPLIT; ++q)
      all &= agree[q];
    if (!all)
      break; // the same decision in every CTA of the cluster
    asm volatile("fence.proxy.async;" ::: "memory"); // the copies below read what other SMs wrote
    pair_step<SORT, ACCV, NSPLIT, UpdBuffers<NSPLIT>::value>(P, step, pair, rank, sm);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0u) {
      __threadfence();
      atomicAdd(P.ver + iB, 1u);
      atomicAdd(P.ver + jB, 1u);
      inval_bars(bars);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// U = G diag(1/||g_c||), D_c = +-||g_c||^2 (share/device_code_common.hpp:187-219)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) initD_kernel(double *const G, double *const D, const unsigned nrow,
                                                    const unsigned ncol, const unsigned nplus, const unsigned ldG)
{
  const unsigned c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const unsigned l = threadIdx.x & 31u;
  if (c >= ncol)
    return;
  double *const g = G + (size_t)c * ldG;
  double x = +0.0;
  for (unsigned r = l; r < nrow; r += 32u) {
    const double y = g[r];
    x = __fma_rn(y, y, x);
  }
  const double y = sum32(x);
  const double nrm = __dsqrt_rn(y);
  for (unsigned r = l; r < nrow; r += 32u)
    g[r] = __ddiv_rn(g[r], nrm);
  if (!l)
    D[c] = (c < nplus) ? y : -y;
}

__global__ void initV_kernel(double *const V, const unsigned ncol, const unsigned ldV)
{
  const size_t n = (size_t)ncol * ncol;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const unsigned c = (unsigned)(i / ncol), r = (unsigned)(i % ncol);
    V[(size_t)c * ldV + r] = (r == c) ? 1.0 : 0.0;
  }
}

// The failure path of the bounded waits, exercised on purpose: each CTA
// waits on an mbarrier that expects one arrival nobody makes, with the given
// cycle limit, records whether the wait gave up and in how many cycles, and
// invalidates the barrier.  Nothing faults or hangs; the context stays usable.
__global__ void wait_selftest_kernel(const long long limit, int *const timed_out, long long *const cycles)
{
  __shared__ uint64_t bar;
  if (threadIdx.x == 0u) {
    mbar_init(&bar, 1u);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0u) {
    const long long t0 = clock64();
    const bool ok = mbar_wait_bounded(&bar, 0u, limit);
    cycles[blockIdx.x] = clock64() - t0;
    if (!ok)
      atomicAdd(timed_out, 1);
    mbar_inval(&bar);
  }
}

// uniform values in (-1, 1) from a counter hash (splitmix64), for the
// autotuner's timed runs
__global__ void fill_random_kernel(double *const a, const size_t n, const unsigned long long seed)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    unsigned long long z = seed + 0x9e3779b97f4a7c15ull * (i + 1u);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    a[i] = (double)(long long)(z >> 11) * 0x1.0p-52 - 1.0;
  }
}

__global__ void rsqrt_test_kernel(const double *const in, double *const out, const unsigned n)
{
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    out[i] = rsqrt_rn(in[i]);
}

__global__ void exact_ops_test_kernel(const unsigned op, const double *const h, const double *const a,
                                      double *const out, int *const ok, const unsigned n)
{
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  bool p;
  switch (op) {
  case 0u:
    out[i] = div_try(h[i], a[i], p);
    break;
  case 1u:
    out[i] = rcp_try(a[i], p);
    break;
  case 2u:
    out[i] = sqrt_try(a[i], p);
    break;
  case 3u:
    out[i] = rsqrt_try(a[i], p);
    break;
  default:
    out[i] = rsqrt_near1(1.0 - a[i], p);
  }
  ok[i] = p ? 1 : 0;
}

// ---------------------------------------------------------------------------
// launchers and tensor maps
// ---------------------------------------------------------------------------
cudaError_t make_update_map(CUtensorMap *tm, const double *base, const unsigned nrow, const unsigned ncol,
                            const unsigned ld)
{
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess)
      return e;
    if (q != cudaDriverEntryPointSuccess || !fn)
      return cudaErrorNotSupported;
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  // (rows within a 32-row piece, pieces, columns); box {34, 8, 16}
  const cuuint64_t dims[3] = {32u, nrow / 32u, ncol};
  const cuuint64_t strides[2] = {32u * sizeof(double), (cuuint64_t)ld * sizeof(double)};
  const cuuint32_t box[3] = {34u, 8u, 16u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3u, const_cast<double *>(base), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t make_gram_map(CUtensorMap *tm, const double *base, const unsigned nrow, const unsigned ncol,
                          const unsigned ld)
{
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess)
      return e;
    if (q != cudaDriverEntryPointSuccess || !fn)
      return cudaErrorNotSupported;
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  // (rows within a 64-row tile, tiles, columns); box {66, 1, 16}
  const cuuint64_t dims[3] = {64u, nrow / 64u, ncol};
  const cuuint64_t strides[2] = {64u * sizeof(double), (cuuint64_t)ld * sizeof(double)};
  const cuuint32_t box[3] = {66u, 1u, 16u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3u, const_cast<double *>(base), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? cudaSuccess : cudaErrorInvalidValue;
}

template <bool S, bool A, unsigned N> static cudaError_t set_smem(const int bytes)
{
  return cudaFuncSetAttribute(l1_step_kernel<S, A, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <bool S, bool A> static cudaError_t set_smem2()
{
  return cudaFuncSetAttribute(l1_step2_kernel<S, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)batch2_smem_bytes());
}

template <bool S, bool A, unsigned F> static cudaError_t set_smem_var(const int bytes)
{
  return cudaFuncSetAttribute(l1_var_kernel<S, A, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

cudaError_t l1_configure()
{
  const int b = (int)l1_smem_bytes();
  cudaError_t e;
  if ((e = set_smem_var<false, false, 1u>(b)) || (e = set_smem_var<false, true, 1u>(b)) ||
      (e = set_smem_var<true, false, 1u>(b)) || (e = set_smem_var<true, true, 1u>(b)) ||
      (e = set_smem_var<false, false, 2u>(b)) || (e = set_smem_var<false, true, 2u>(b)) ||
      (e = set_smem_var<true, false, 2u>(b)) || (e = set_smem_var<true, true, 2u>(b)))
    return e;
  if ((e = set_smem2<false, false>()) || (e = set_smem2<false, true>()) || (e = set_smem2<true, false>()) ||
      (e = set_smem2<true, true>()))
    return e;
  const int bu = (int)(kUSmemDoubles * sizeof(double)), bn = (int)batchn_smem_bytes();
  constexpr auto kSmem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((e = cudaFuncSetAttribute(l1_update_kernel<false>, kSmem, bu)) ||
      (e = cudaFuncSetAttribute(l1_update_kernel<true>, kSmem, bu)) ||
      (e = cudaFuncSetAttribute(l1_stepn_kernel<false>, kSmem, bn)) ||
      (e = cudaFuncSetAttribute(l1_stepn_kernel<true>, kSmem, bn)))
    return e;
  const int b3 = (int)step_smem_bytes(2u);
  if ((e = set_smem<false, false, 1u>(b)) || (e = set_smem<false, true, 1u>(b)) || (e = set_smem<true, false, 1u>(b)) ||
      (e = set_smem<true, true, 1u>(b)) || (e = set_smem<false, false, 2u>(b3)) || (e = set_smem<false, true, 2u>(b3)) ||
      (e = set_smem<true, false, 2u>(b3)) || (e = set_smem<true, true, 2u>(b3)) ||
      (e = set_smem<false, false, 4u>(b3)) || (e = set_smem<false, true, 4u>(b3)) ||
      (e = set_smem<true, false, 4u>(b3)) || (e = set_smem<true, true, 4u>(b3)) ||
      (e = set_smem<false, false, 8u>(b3)) || (e = set_smem<false, true, 8u>(b3)) ||
      (e = set_smem<true, false, 8u>(b3)) || (e = set_smem<true, true, 8u>(b3)))
    return e;
  return cudaSuccess;
}

template <bool S, bool A, unsigned N> static cudaError_t launch(const StepParams &p, cudaStream_t s)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.pairs * N);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = step_smem_bytes(N);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = N;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, l1_step_kernel<S, A, N>, p);
}

template <bool S, bool A, unsigned N> static cudaLaunchConfig_t sweep_cfg(const StepParams &p, cudaStream_t s,
                                                                         cudaLaunchAttribute *at)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.pairs * N);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = step_smem_bytes(N);
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = N;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeCooperative;
  at[1].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cfg;
}

template <bool S, bool A, unsigned N> static bool sweep_fits(const StepParams &p)
{
  if (cudaFuncSetAttribute(l1_sweep_kernel<S, A, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)step_smem_bytes(N)) != cudaSuccess)
    return false;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = sweep_cfg<S, A, N>(p, nullptr, at);
  cfg.numAttrs = 1; // the occupancy query takes the cluster shape
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, l1_sweep_kernel<S, A, N>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return (unsigned)clusters >= p.pairs;
}

template <bool S, bool A, unsigned N> static cudaError_t sweep_launch(const StepParams &p, cudaStream_t s)
{
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = sweep_cfg<S, A, N>(p, s, at);
  return cudaLaunchKernelEx(&cfg, l1_sweep_kernel<S, A, N>, p);
}

bool sweep_kernel_fits(const bool sort, const bool accv, const StepParams &p)
{
  if (p.split > 4u) // clusters of 8: one launch per step only
    return false;
  if (p.split == 4u) {
    if (sort)
      return accv ? sweep_fits<true, true, 4u>(p) : sweep_fits<true, false, 4u>(p);
    return accv ? sweep_fits<false, true, 4u>(p) : sweep_fits<false, false, 4u>(p);
  }
  if (p.split == 2u) {
    if (sort)
      return accv ? sweep_fits<true, true, 2u>(p) : sweep_fits<true, false, 2u>(p);
    return accv ? sweep_fits<false, true, 2u>(p) : sweep_fits<false, false, 2u>(p);
  }
  if (sort)
    return accv ? sweep_fits<true, true, 1u>(p) : sweep_fits<true, false, 1u>(p);
  return accv ? sweep_fits<false, true, 1u>(p) : sweep_fits<false, false, 1u>(p);
}

cudaError_t launch_l1_sweep(const bool sort, const bool accv, const StepParams &p, cudaStream_t s)
{
  if (p.split == 4u) {
    if (sort)
      return accv ? sweep_launch<true, true, 4u>(p, s) : sweep_launch<true, false, 4u>(p, s);
    return accv ? sweep_launch<false, true, 4u>(p, s) : sweep_launch<false, false, 4u>(p, s);
  }
  if (p.split == 2u) {
    if (sort)
      return accv ? sweep_launch<true, true, 2u>(p, s) : sweep_launch<true, false, 2u>(p, s);
    return accv ? sweep_launch<false, true, 2u>(p, s) : sweep_launch<false, false, 2u>(p, s);
  }
  if (sort)
    return accv ? sweep_launch<true, true, 1u>(p, s) : sweep_launch<true, false, 1u>(p, s);
  return accv ? sweep_launch<false, true, 1u>(p, s) : sweep_launch<false, false, 1u>(p, s);
}

// The largest clusters that are all resident at once, 8 CTAs only from this many
// rows: below, their thinner Gram shares and fewer update stages do not pay for
// the wider exchange.  us per call of n = 256, ALG 11, with 8 / 4 CTAs per pair:
// 256 rows 5256 / 5247, 512: 5470 / 5483, 1024: 5935 / 6444, 4096: 9394 / 10813,
// 16384: 22471 / 28281.  us per sweep of other column counts (ALG 9): 1024 rows
// x 32: 86 / 87, x 64: 150 / 153, x 128: 292 / 296, x 192: 435 / 442, x 320: 717 / 735, x
// 448: 1001 / 1026; 8192 rows: 221 / 233, 383 / 422, 709 / 809, 1084 / 1231, 1831 /
// 2090, 2537 / 3007; 512 rows: within 3 % either way.  More clusters than fit at
// once run in two waves: 34 pairs per step (2048 x 1088) take 104 ms with 4 CTAs
// per pair, 67 ms with 2; 16 pairs (1024 x 512) 2.05 ms a sweep with 8, 1.17 with 4.
constexpr unsigned kSplit8Rows = 1024u;

// how many clusters of N CTAs of the step kernel the current device holds at
// once (a GPC's SMs divide into whole clusters only, so fewer than SMs / N)
template <unsigned N> static unsigned resident_clusters()
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(N);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = step_smem_bytes(N);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = N;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, l1_step_kernel<true, true, N>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0u;
  }
  return (unsigned)n;
}

unsigned l1_split(const unsigned pairs, const unsigned nrow)
{
  struct Fit {
    bool known = false;
    unsigned c8 = 0u, c4 = 0u, c2 = 0u;
  };
  static Fit fits[64]; // by device; the caller holds the library's lock
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64)
    return 1u;
  Fit &f = fits[dev];
  if (!f.known)
    f = Fit{true, resident_clusters<8u>(), resident_clusters<4u>(), resident_clusters<2u>()};
  if (pairs <= f.c8 && nrow >= kSplit8Rows)
    return 8u;
  return (pairs <= f.c4) ? 4u : (pairs <= f.c2) ? 2u : 1u;
}

// a launch that may be placed before the one before it in the stream is complete
template <typename K>
static cudaError_t launch_pdl(K *const kernel, const unsigned ctas, const unsigned threads, const size_t smem,
                              const StepParams &p, cudaStream_t s)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <bool S, bool A> static cudaError_t launch2(const StepParams &p, cudaStream_t s)
{
  return launch_pdl(l1_step2_kernel<S, A>, (p.pairs + 1u) / 2u, kThreads, batch2_smem_bytes(), p, s);
}

template <bool S, bool A, unsigned F> static cudaError_t launch_var(const StepParams &p, cudaStream_t s)
{
  l1_var_kernel<S, A, F><<<p.pairs, kThreads, l1_smem_bytes(), s>>>(p);
  return cudaGetLastError();
}

// the block pairs of a step up to their transforms (p.vt), by the step kernels
// without V (they leave before the update)
static cudaError_t launch_factor(const bool sort, const StepParams &p, cudaStream_t s)
{
  if (p.width == kWidthHalf) {
    return launch_pdl(sort ? l1_stepn_kernel<true> : l1_stepn_kernel<false>, p.pairs, kNThreads, batchn_smem_bytes(), p,
                      s);
  }
  switch (p.split) {
  case 8u:
    return sort ? launch<true, false, 8u>(p, s) : launch<false, false, 8u>(p, s);
  case 4u:
    return sort ? launch<true, false, 4u>(p, s) : launch<false, false, 4u>(p, s);
  case 2u:
    return sort ? launch<true, false, 2u>(p, s) : launch<false, false, 2u>(p, s);
  default:
    return sort ? launch<true, false, 1u>(p, s) : launch<false, false, 1u>(p, s);
  }
}

template <bool A> static cudaError_t launch_update(const StepParams &p, cudaStream_t s)
{
  const unsigned nst = (p.nrow + kUpdRows - 1u) / kUpdRows + (A ? (p.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  const unsigned total = p.pairs * nst;
  return launch_pdl(l1_update_kernel<A>, total < p.sms ? total : p.sms, kThreads, kUSmemDoubles * sizeof(double), p, s);
}

cudaError_t launch_l1_step(const bool sort, const bool accv, const StepParams &p, cudaStream_t s)
{
  if (p.variant == 1u) {
    if (sort)
      return accv ? launch_var<true, true, 1u>(p, s) : launch_var<true, false, 1u>(p, s);
    return accv ? launch_var<false, true, 1u>(p, s) : launch_var<false, false, 1u>(p, s);
  }
  if (p.variant == 2u) {
    if (sort)
      return accv ? launch_var<true, true, 2u>(p, s) : launch_var<true, false, 2u>(p, s);
    return accv ? launch_var<false, true, 2u>(p, s) : launch_var<false, false, 2u>(p, s);
  }
  if (p.vt) {
    const cudaError_t e = launch_factor(sort, p, s);
    return (e != cudaSuccess) ? e : (accv ? launch_update<true>(p, s) : launch_update<false>(p, s));
  }
  const unsigned n = p.split;
  if (n == 1u && p.width == 2u) {
    if (sort)
      return accv ? launch2<true, true>(p, s) : launch2<true, false>(p, s);
    return accv ? launch2<false, true>(p, s) : launch2<false, false>(p, s);
  }
  if (n == 8u) {
    if (sort)
      return accv ? launch<true, true, 8u>(p, s) : launch<true, false, 8u>(p, s);
    return accv ? launch<false, true, 8u>(p, s) : launch<false, false, 8u>(p, s);
  }
  if (n == 4u) {
    if (sort)
      return accv ? launch<true, true, 4u>(p, s) : launch<true, false, 4u>(p, s);
    return accv ? launch<false, true, 4u>(p, s) : launch<false, false, 4u>(p, s);
  }
  if (n == 2u) {
    if (sort)
      return accv ? launch<true, true, 2u>(p, s) : launch<true, false, 2u>(p, s);
    return accv ? launch<false, true, 2u>(p, s) : launch<false, false, 2u>(p, s);
  }
  if (sort)
    return accv ? launch<true, true, 1u>(p, s) : launch<true, false, 1u>(p, s);
  return accv ? launch<false, true, 1u>(p, s) : launch<false, false, 1u>(p, s);
}

cudaError_t launch_initD(double *G, double *D, unsigned nrow, unsigned ncol, unsigned nplus, unsigned ldG,
                         cudaStream_t s)
{
  const unsigned wpb = 8u;
  initD_kernel<<<(ncol + wpb - 1u) / wpb, 32u * wpb, 0, s>>>(G, D, nrow, ncol, nplus, ldG);
  return cudaGetLastError();
}

cudaError_t launch_initV(double *V, unsigned ncol, unsigned ldV, cudaStream_t s)
{
  const size_t n = (size_t)ncol * ncol;
  unsigned blocks = (unsigned)((n + 255u) / 256u);
  if (blocks > 4096u)
    blocks = 4096u;
  initV_kernel<<<blocks, 256u, 0, s>>>(V, ncol, ldV);
  return cudaGetLastError();
}

cudaError_t launch_wait_selftest(long long limit, int *timed_out, long long *cycles, unsigned ctas, cudaStream_t s)
{
  wait_selftest_kernel<<<ctas, 32u, 0, s>>>(limit, timed_out, cycles);
  return cudaGetLastError();
}

cudaError_t launch_fill_random(double *a, size_t n, unsigned long long seed, cudaStream_t s)
{
  fill_random_kernel<<<1024u, 256u, 0, s>>>(a, n, seed);
  return cudaGetLastError();
}

cudaError_t launch_exact_ops_test(unsigned op, const double *h, const double *a, double *out, int *ok, unsigned n,
                                  cudaStream_t s)
{
  exact_ops_test_kernel<<<(n + 255u) / 256u, 256u, 0, s>>>(op, h, a, out, ok, n);
  return cudaGetLastError();
}

cudaError_t launch_rsqrt_test(const double *in, double *out, unsigned n, cudaStream_t s)
{
  rsqrt_test_kernel<<<(n + 255u) / 256u, 256u, 0, s>>>(in, out, n);
  return cudaGetLastError();
}

} // namespace gjx
