// gjx_batch.cu -- the batched form, one launch per outer step index.
#include "gjx_pair.cuh"

namespace gjx {

// ---------------------------------------------------------------------------
// Batched form: each launch advances every active matrix of a batch by one
// outer step of its own sweep (matrix b: step kstep[b] mod steps1), so small
// matrices run their short sweeps back to back while large ones progress.  A
// persistent grid (one CTA per SM) takes the block pairs -- (matrix << 16) |
// pair, largest matrices first -- from a work queue, W at a time: with W = 2
// two live pairs go through pair_step2 together, a lone one through
// pair_step with one CTA, so every matrix gets the bits it would get alone.
// Converged matrices are skipped.  The mbarriers are invalidated after each
// item (both step forms initialise them).
// ---------------------------------------------------------------------------
template <bool SORT, bool ACCV, unsigned W>
__global__ void __launch_bounds__(kThreads, 1) l1_batch_kernel(const __grid_constant__ BatchStep B)
{
  extern __shared__ __align__(128) double sm[];
  __shared__ unsigned item;
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kOffBar);
  for (;;) {
    if (threadIdx.x == 0u)
      item = atomicAdd(B.queue, W);
    __syncthreads();
    const unsigned it = item;
    const bool stop = (it >= B.nitems) || (*(volatile int *)B.err != 0);
    __syncthreads(); // every thread has read item
    if (stop)
      break;
    const uint32_t e0 = B.items[it];
    const unsigned b0 = e0 >> 16u;
    const bool live0 = !B.done[b0];
    uint32_t e1 = 0u;
    bool live1 = false;
    if (W == 2u && it + 1u < B.nitems) {
      e1 = B.items[it + 1u];
      live1 = !B.done[e1 >> 16u];
    }
    if (!live0 && !live1)
      continue;
    if (live0 && live1 && B.mats[b0].p.strat0 == B.mats[e1 >> 16u].p.strat0) {
      const BatchMat &ma = B.mats[b0], &mb = B.mats[e1 >> 16u];
      pair_step2<SORT, ACCV>(ma.p, B.kstep[b0] % ma.steps1, e0 & 0xffffu, mb.p, B.kstep[e1 >> 16u] % mb.steps1,
                             e1 & 0xffffu, sm);
    }
    else {
      for (unsigned h = 0u; h < 2u; ++h) {
        const bool live = h ? live1 : live0;
        if (!live)
          continue;
        const uint32_t e = h ? e1 : e0;
        const BatchMat &m = B.mats[e >> 16u];
        pair_step<SORT, ACCV, 1u>(m.p, B.kstep[e >> 16u] % m.steps1, e & 0xffffu, 0u, sm);
        __syncthreads();
        if (threadIdx.x == 0u)
          inval_bars(bars);
        __syncthreads();
      }
      continue;
    }
    __syncthreads();
    if (threadIdx.x == 0u)
      inval_bars(bars);
    __syncthreads();
  }
}

// The batched step on CTAs of 4 warps, two per SM: a CTA takes one block pair
// at a time from the queue (the same queue, items and skips as
// l1_batch_kernel).  The mbarriers are invalidated after each item.
template <bool SORT, bool ACCV>
__global__ void __launch_bounds__(kNThreads, 2) l1_batchn_kernel(const __grid_constant__ BatchStep B)
{
  extern __shared__ __align__(128) double sm[];
  __shared__ unsigned item;
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kNOffBar);
  for (;;) {
    if (threadIdx.x == 0u)
      item = atomicAdd(B.queue, 1u);
    __syncthreads();
    const unsigned it = item;
    const bool stop = (it >= B.nitems) || (*(volatile int *)B.err != 0);
    __syncthreads(); // every thread has read item
    if (stop)
      break;
    const uint32_t e = B.items[it];
    const unsigned b = e >> 16u;
    if (B.done[b])
      continue;
    const BatchMat &m = B.mats[b];
    pair_step_n<SORT, ACCV>(m.p, B.kstep[b] % m.steps1, e & 0xffffu, sm);
    __syncthreads();
    if (threadIdx.x == 0u)
      inval_bars_n(bars);
    __syncthreads();
  }
}

// The batched step on CTAs of 4 warps, two per SM, two block pairs per CTA
// at a time (items taken in twos from the queue, as l1_batch_kernel with W =
// 2): two live pairs with the same inner table through pair_step2n, a lone
// one through pair_step_n.  The mbarriers are invalidated after each item.
template <bool SORT, bool ACCV>
__global__ void __launch_bounds__(kNThreads, 2) l1_batchn2_kernel(const __grid_constant__ BatchStep B)
{
  extern __shared__ __align__(128) double sm[];
  __shared__ unsigned item;
  auto inval = [&](uint64_t *const bars) {
    __syncthreads();
    if (threadIdx.x == 0u)
      inval_bars_n(bars);
    __syncthreads();
  };
  for (;;) {
    if (threadIdx.x == 0u)
      item = atomicAdd(B.queue, 2u);
    __syncthreads();
    const unsigned it = item;
    const bool stop = (it >= B.nitems) || (*(volatile int *)B.err != 0);
    __syncthreads(); // every thread has read item
    if (stop)
      break;
    const uint32_t e0 = B.items[it];
    const bool live0 = !B.done[e0 >> 16u];
    uint32_t e1 = 0u;
    bool live1 = false;
    if (it + 1u < B.nitems) {
      e1 = B.items[it + 1u];
      live1 = !B.done[e1 >> 16u];
    }
    if (live0 && live1 && B.mats[e0 >> 16u].p.strat0 == B.mats[e1 >> 16u].p.strat0) {
      const BatchMat &ma = B.mats[e0 >> 16u], &mb = B.mats[e1 >> 16u];
      pair_step2n<SORT, ACCV>(ma.p, B.kstep[e0 >> 16u] % ma.steps1, e0 & 0xffffu, mb.p,
                              B.kstep[e1 >> 16u] % mb.steps1, e1 & 0xffffu, sm);
      inval(reinterpret_cast<uint64_t *>(sm + kN2OffBar));
      continue;
    }
    for (unsigned h = 0u; h < 2u; ++h) {
      if (!(h ? live1 : live0))
        continue;
      const uint32_t e = h ? e1 : e0;
      const BatchMat &m = B.mats[e >> 16u];
      pair_step_n<SORT, ACCV>(m.p, B.kstep[e >> 16u] % m.steps1, e & 0xffffu, sm);
      inval(reinterpret_cast<uint64_t *>(sm + kNOffBar));
    }
  }
}

// after a launch of the batch: one step more for every active matrix; at the
// end of its sweep, its totals and the convergence test (no big rotation in
// the sweep, or the sweep cap); the work queue cleared for the next launch
__global__ void batch_sweep_end_kernel(const BatchSweep S)
{
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0u)
    S.queue[0] = 0u;
  if (i >= S.nmat || S.done[i])
    return;
  const unsigned k = ++S.kstep[i];
  if (k % S.mats[i].steps1) { // the sweep goes on
    atomicAdd(S.active, 1u);
    return;
  }
  const unsigned long long c = S.cvg[i];
  S.cvg[i] = 0ull;
  const unsigned small = (unsigned)c, big = (unsigned)(c >> 32u);
  S.glb_s[i] += small;
  S.glb_b[i] += big;
  const unsigned sw = ++S.sweeps[i];
  if (!big || sw >= kNSweep)
    S.done[i] = 1u;
  else
    atomicAdd(S.active, 1u);
}

// initD for a batch: block b normalises the columns of matrix b, one warp
// per column, the same arithmetic as initD_kernel
__global__ void __launch_bounds__(256) initD_batch_kernel(const BatchMat *const M, const unsigned nmat,
                                                          const uint32_t *const done_ok)
{
  const BatchMat &m = M[blockIdx.x];
  if (blockIdx.x >= nmat || !done_ok[blockIdx.x])
    return;
  const unsigned l = threadIdx.x & 31u;
  for (unsigned c = threadIdx.x >> 5; c < m.p.ncol; c += blockDim.x >> 5) {
    double *const g = m.p.G + (size_t)c * m.p.ldG;
    double x = +0.0;
    for (unsigned r = l; r < m.p.nrow; r += 32u) {
      const double y = g[r];
      x = __fma_rn(y, y, x);
    }
    const double y = sum32(x);
    const double nrm = __dsqrt_rn(y);
    for (unsigned r = l; r < m.p.nrow; r += 32u)
      g[r] = __ddiv_rn(g[r], nrm);
    if (!l)
      m.D[c] = (c < m.p.nplus) ? y : -y;
  }
}

__global__ void initV_batch_kernel(const BatchMat *const M, const unsigned nmat)
{
  for (unsigned b = blockIdx.y; b < nmat; b += gridDim.y) {
    const BatchMat &m = M[b];
    if (!m.p.V)
      continue;
    const size_t n = (size_t)m.p.ncol * m.p.ncol;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
      const unsigned c = (unsigned)(i / m.p.ncol), r = (unsigned)(i % m.p.ncol);
      m.p.V[(size_t)c * m.p.ldV + r] = (r == c) ? 1.0 : 0.0;
    }
  }
}

template <bool S, bool A> static cudaError_t set_smem_batch()
{
  cudaError_t e = cudaFuncSetAttribute(l1_batch_kernel<S, A, 1u>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)l1_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(l1_batch_kernel<S, A, 2u>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)batch2_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(l1_batchn_kernel<S, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)batchn_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(l1_batchn2_kernel<S, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)batchn2_smem_bytes());
  return e;
}

cudaError_t batch_configure()
{
  cudaError_t e;
  if ((e = set_smem_batch<false, false>()) || (e = set_smem_batch<false, true>()) ||
      (e = set_smem_batch<true, false>()) || (e = set_smem_batch<true, true>()))
    return e;
  return cudaSuccess;
}

template <bool S, bool A>
static void batch_launch(const unsigned width, const BatchStep &b, const unsigned ctas, cudaStream_t s)
{
  if (width == kWidthHalf)
    l1_batchn_kernel<S, A><<<ctas, kNThreads, batchn_smem_bytes(), s>>>(b);
  else if (width == kWidthHalf2)
    l1_batchn2_kernel<S, A><<<ctas, kNThreads, batchn2_smem_bytes(), s>>>(b);
  else if (width == 2u)
    l1_batch_kernel<S, A, 2u><<<ctas, kThreads, batch2_smem_bytes(), s>>>(b);
  else
    l1_batch_kernel<S, A, 1u><<<ctas, kThreads, l1_smem_bytes(), s>>>(b);
}

cudaError_t launch_batch_step(const bool sort, const bool accv, const unsigned width, const BatchStep &b,
                              const unsigned ctas, cudaStream_t s)
{
  if (sort) {
    if (accv)
      batch_launch<true, true>(width, b, ctas, s);
    else
      batch_launch<true, false>(width, b, ctas, s);
  }
  else if (accv)
    batch_launch<false, true>(width, b, ctas, s);
  else
    batch_launch<false, false>(width, b, ctas, s);
  return cudaGetLastError();
}

cudaError_t launch_batch_sweep_end(const BatchSweep &w, cudaStream_t s)
{
  batch_sweep_end_kernel<<<(w.nmat + 255u) / 256u, 256u, 0, s>>>(w);
  return cudaGetLastError();
}

cudaError_t launch_batch_initV(const BatchMat *m, unsigned nmat, cudaStream_t s)
{
  initV_batch_kernel<<<dim3(8u, nmat < 4096u ? nmat : 4096u), 256u, 0, s>>>(m, nmat);
  return cudaGetLastError();
}

cudaError_t launch_batch_initD(const BatchMat *m, unsigned nmat, const uint32_t *ok, cudaStream_t s)
{
  initD_batch_kernel<<<nmat, 256u, 0, s>>>(m, nmat, ok);
  return cudaGetLastError();
}

} // namespace gjx
