// gjx_pair.cuh -- the block-pair step of the blocked one-sided Jacobi (H)SVD
// (sm_100a device code of the plain form; the kernels are in gjx_kernels.cu,
// gjx_batch.cu and gjx_flow.cu).
//
// One block pair (i, j) of an outer step is processed by a cluster of NSPLIT
// CTAs (NSPLIT = 8, 4 or 2 when the step has few pairs, so that more SMs work on
// each pair; 1 when the pairs already fill the GPU), 256 threads each:
//
//   1. Gram matrix of the M x 32 column pair [G_i G_j], lower triangle only
//      (the Cholesky never reads the upper one).  Each CTA streams the whole
//      pair through shared memory in 64-row tiles (TMA tensor copies into a
//      bank-skewed, zero-padded layout, mbarrier completion, 4 stages of 2
//      tiles) and computes its share of the 528 entries; every
//      entry is one FMA chain in the reference's row order
//      (share/device_code_common_Cholesky.hpp:4-56).  A lane holds 1 (8-CTA
//      clusters) to 8 chains (one CTA per pair) of neighbouring columns x and
//      one or two columns y.  The shares are exchanged through distributed shared memory,
//      then one cluster barrier.
//   2. 32x32 Cholesky by two warps, the trailing matrix in registers
//      (share/device_code_common_Cholesky.hpp:58-158).
//   3. Inner Jacobi sweep(s) on R: per inner step 16 lanes take each of the 16
//      column pairs, sum its dot products in the reference's order, evaluate
//      its rotation (branch-free; trigonometric or hyperbolic, optional KISS
//      sorting) and apply it to their two rows of R and V_loc; one barrier per
//      step (share/device_code_nosort.hpp, share/device_code_cdsort.hpp,
//      share/device_code_cdsort_KISS.hpp).
//      Steps 2 and 3 are deterministic, so every CTA of the cluster computes
//      them itself and holds the same V_loc bit for bit.
//   4. [G_i G_j] <- [G_i G_j] V_loc (and V likewise): 256-row stages brought
//      in by TMA tensor copies, the stages dealt out to the CTAs of the
//      cluster (the first one in flight during steps 2 and 3); each output
//      is a 32-FMA chain in the reference's skewed order
//      (share/device_code_common.hpp:146-185), computed in 4x8 register
//      tiles along anti-diagonals, put back in place of the stage's operands
//      and written out by TMA tensor stores that overlap the next stage.
//
// pair_step2 runs two block pairs in one CTA (the batched form, and steps
// with more pairs than SMs): steps 1 and 4 of the two one after the other on
// all warps, steps 2 and 3 concurrently on two groups of 4 warps.
//
// All arithmetic is in the reference's order, so results are bit-identical.
#pragma once

#include <cooperative_groups.h>

#include "gjx_device.cuh"
#include "gjx_internal.h"
#include "gjx_qr.cuh"

namespace cg = cooperative_groups;

namespace gjx {

constexpr unsigned kThreads = 256u;
constexpr long long kWaitLimit = 2000000000ll; // ~1 s of cycles per wait

// Gram staging: a stage holds 2 tiles of 64 rows of the 32 columns, brought
// in by the TMA engine: per tile and block one box {66 rows, 1 tile, 16
// columns} of the 3-D view (64 rows, tiles, columns) of G.  Rows 64-65 lie
// outside the view and are zero-filled, so column c of a tile starts at
// c * 66.  The column stride of 66 doubles (33 16-byte granules, odd) puts the
// row pairs of 8 consecutive columns in 8 bank groups.  4 stages in flight;
// the copies are issued by a thread of warp 7, which computes no Gram entry.
constexpr unsigned kGramTiles = 2u;
constexpr unsigned kGramStages = 4u;
constexpr unsigned kGramColLd = 66u;
constexpr unsigned kGramTileLd = 32u * kGramColLd;
constexpr unsigned kGramStage = kGramTiles * kGramTileLd; // doubles
constexpr uint32_t kGramBoxBytes = 66u * 16u * 8u;
constexpr unsigned kIssuer = 224u; // lane 0 of warp 7

// Update staging: 256 rows x 32 columns; the 32-row piece p of column c
// starts at c*272 + p*34 (2 doubles of skew per piece spread the banks).
// One TMA tensor copy per block and stage: a 3-D view (32 rows, pieces,
// columns) of the matrix and a box of {34, 8, 16} lands exactly in this
// layout (rows 32 and 33 of a piece box lie outside the view: zero fill).
constexpr unsigned kUpdRows = 256u;
constexpr unsigned kUpdColLd = 272u;
constexpr unsigned kUpdStages = 2u;
constexpr unsigned kUpdStage = 32u * kUpdColLd; // doubles
constexpr unsigned kVTLd = 34u;                 // B^T rows (V_loc transposed)
static_assert(kTransform == 32u * kVTLd, "the layout of StepParams::vt");
constexpr uint32_t kUpdBoxBytes = 34u * 8u * 16u * 8u;

constexpr unsigned kRegion =
    (kGramStages * kGramStage > kUpdStages * kUpdStage) ? kGramStages * kGramStage : kUpdStages * kUpdStage;

// shared memory map (in doubles)
constexpr unsigned kOffR = kRegion;        // R, 32x32 (later B^T, 32x34)
constexpr unsigned kOffVl = kOffR + 32u * kVTLd;
constexpr unsigned kOffS0 = kOffVl + 1024u; // strat0 copy, 1024 bytes
constexpr unsigned kOffRed = kOffS0 + 128u; // 32 unsigned
constexpr unsigned kOffBar = kOffRed + 16u; // mbarriers: [0..3] Gram stages, [4..6] update stages landed,
                                            // [8..10] update stages done (one arrival per warp),
                                            // [11..14] Gram stages read (one arrival per Gram warp)
constexpr unsigned kBars = 15u;
constexpr unsigned kGramWarps = 3u; // warps 0-2 compute Gram entries
constexpr unsigned kSmemDoubles = kOffBar + 16u;

// every step form of 8 warps starts with all of them initialised
__device__ __forceinline__ void init_bars(uint64_t *const bars)
{
  for (unsigned b = 0u; b < kBars; ++b)
    mbar_init(&bars[b], (b < 8u) ? 1u : (b < 11u) ? kThreads / 32u : kGramWarps); // < 8: the expected bytes
  mbar_fence_init();
}

__device__ __forceinline__ void inval_bars(uint64_t *const bars)
{
  for (unsigned b = 0u; b < kBars; ++b)
    mbar_inval(&bars[b]);
}

inline size_t l1_smem_bytes() { return (size_t)kSmemDoubles * sizeof(double); }

// the step kernels of clusters keep a third update buffer after
// the rest (128-byte aligned), 227 KB in all
constexpr unsigned kOffUpd3 = (kSmemDoubles + 15u) & ~15u;
constexpr unsigned kSmemDoubles3 = kOffUpd3 + kUpdStage;
static_assert(kSmemDoubles3 * sizeof(double) <= 227u * 1024u, "the third update buffer must fit");
template <unsigned NSPLIT> struct UpdBuffers {
  static constexpr unsigned value = (NSPLIT > 1u) ? 3u : 2u;
};
inline size_t step_smem_bytes(const unsigned nsplit)
{
  return (size_t)((nsplit > 1u) ? kSmemDoubles3 : kSmemDoubles) * sizeof(double);
}

#define E32(A, r, c) (A)[(c) * 32u + (r)]

// ---------------------------------------------------------------------------
// Gram: one 64-row tile for the XU YU chains (x, y) of a lane, x = X0 + lx XU + u
// (u < XU), y = y0 + v dy (v < YU).  Chain (x, y) adds G[r,y]*G[r,x] for r = x,
// x+1, ..., x+63 (mod 64), the reference's order.  With k = r - X0 the chain
// takes the k in [d, d+63], d = lx XU + u, in increasing order (rows mod 64); lx
// is below LX (1 or 2), so a block's lanes read the same rows in the same
// iteration and differ only in the first and last LX XU of them.
// Operands come in 16-byte pairs of rows (k, k+1), k even, the pairs of k + 4
// in flight while those of k are used.
// What bounds it (measured on resident operands): a sub-partition takes in one
// 16-byte load of a warp in 7 to 8 cycles whatever its addresses, the SM one
// distinct 128 bytes per half-warp in a cycle, and a chain one FMA in 9.7.  So
// in the clusters a lane holds few chains of many operands shared, and lanes
// 2j, 2j+1 share their columns y, all even (odd) lanes their columns x: 8
// columns y per half-warp, in 8 bank groups.  Cycles per tile of the 3 warps of
// a CTA: 1x1 649 (8 CTAs), 1x2 768 (4 CTAs), 2x2 1093 (2 CTAs); before, with 32
// columns y per warp, 2x1 864 (4 CTAs) and 4x1 1306 (2 CTAs).  With one CTA per
// pair the chains fill 3 warps best as 4x2 with LX = 1 (1779; 2x2 on 4 warps
// with the diagonal blocks beside other chains measured 25 % slower).
// ---------------------------------------------------------------------------
template <unsigned XU, unsigned YU, unsigned LX>
__device__ __forceinline__ void gram_tile(const double *const st, const unsigned X0, const unsigned lx,
                                          const unsigned y0, const unsigned dy, double (&acc)[XU][YU])
{
  constexpr unsigned NP = (64u + LX * XU) / 2u; // row pairs: k = 0 .. 63 + LX XU - 1
  const double *const yp = st + y0 * kGramColLd;
  const double *const xp = st + (X0 + lx * XU) * kGramColLd;
  double2 Yb[3][YU], Xb[3][XU];
  const auto load = [&](const unsigned kp) {
    const unsigned q = kp % 3u, o = (X0 + 2u * kp) & 63u;
#pragma unroll
    for (unsigned v = 0u; v < YU; ++v)
      Yb[q][v] = *reinterpret_cast<const double2 *>(yp + v * dy * kGramColLd + o);
#pragma unroll
    for (unsigned u = 0u; u < XU; ++u)
      if (LX > 1u || (2u * kp + 1u >= u && 2u * kp <= u + 63u))
        Xb[q][u] = *reinterpret_cast<const double2 *>(xp + u * kGramColLd + o);
  };
  load(0u);
  load(1u);
#pragma unroll
  for (unsigned kp = 0u; kp < NP; ++kp) { // pairs k = 2kp, 2kp + 1
    if (kp + 2u < NP)
      load(kp + 2u);
    const unsigned q = kp % 3u;
#pragma unroll
    for (unsigned h = 0u; h < 2u; ++h) {
      const unsigned k = 2u * kp + h;
#pragma unroll
      for (unsigned u = 0u; u < XU; ++u) {
        const double xv = h ? Xb[q][u].y : Xb[q][u].x;
        if (k < u || k > (LX - 1u) * XU + u + 63u) // no lane's row
          continue;
        // lx = 0 has begun at k = u and ends at u + 63, lx = 1 XU later
        const bool on = (LX == 1u) ? true : (k < XU + u) ? (lx == 0u) : (k > u + 63u) ? (lx != 0u) : true;
        if (on) {
#pragma unroll
          for (unsigned v = 0u; v < YU; ++v)
            acc[u][v] = __fma_rn(h ? Yb[q][v].y : Yb[q][v].x, xv, acc[u][v]);
        }
      }
    }
  }
}

// The lanes.  x-block b is the rows LX XU b .. LX XU (b + 1) - 1.  It has the
// columns y = 0 .. LX XU (b + 1) - 1 (entries with y > x are computed and
// dropped), nj = LX XU (b + 1) / YU of them with v = 0; its lane LX j + lx takes
// y = j + v nj.  Blocks of the warps:
//   1 CTA: 4x2, LX 1; warps (7, 6, 0), (5, 4, 3), (2, 1): 72 lanes.
//   2 CTAs: 2x2, LX 2; (7), (6, 0), (1) of rank 0, (5), (4, 2), (3) of rank 1:
//     72 lanes.
//   4 CTAs: 1x2, LX 2; (15 - rank), (8 + rank, rank), (7 - rank): 68 lanes.
//   8 CTAs: 1x1, LX 2; block 15 - rank in warps 0 and 1, block rank in warp 2:
//     68 lanes.
template <unsigned NSPLIT> struct GramShape {
  static constexpr unsigned XU = (NSPLIT == 1u) ? 4u : (NSPLIT == 2u) ? 2u : 1u;
  static constexpr unsigned YU = (NSPLIT <= 4u) ? 2u : 1u;
  static constexpr unsigned LX = (NSPLIT == 1u) ? 1u : 2u;
  static constexpr unsigned warps = kGramWarps;
};

struct GramLane {
  unsigned X0, lx, y0, dy;
  bool on;
};

template <unsigned NSPLIT>
__device__ __forceinline__ GramLane gram_lane(const unsigned rank, const unsigned warp, const unsigned lane)
{
  using S = GramShape<NSPLIT>;
  GramLane g = {0u, 0u, 0u, 0u, false};
  if (warp >= S::warps)
    return g;
  int blk[3] = {-1, -1, -1}; // the warp's blocks, in the order of their lanes
  unsigned l = lane;
  if constexpr (NSPLIT == 1u) {
    blk[0] = (warp == 0u) ? 7 : (warp == 1u) ? 5 : 2;
    blk[1] = (warp == 0u) ? 6 : (warp == 1u) ? 4 : 1;
    blk[2] = (warp == 0u) ? 0 : (warp == 1u) ? 3 : -1;
  }
  else if constexpr (NSPLIT == 2u) {
    blk[0] = (rank == 0u) ? ((warp == 2u) ? 1 : 7 - (int)warp) : 5 - (int)warp;
    blk[1] = (warp == 1u) ? (rank == 0u ? 0 : 2) : -1;
  }
  else if constexpr (NSPLIT == 4u) {
    blk[0] = (warp == 0u) ? 15 - (int)rank : (warp == 1u) ? 8 + (int)rank : 7 - (int)rank;
    blk[1] = (warp == 1u) ? (int)rank : -1;
  }
  else {
    blk[0] = (warp < 2u) ? 15 - (int)rank : (int)rank;
    l = (warp == 1u) ? lane + 32u : lane;
  }
#pragma unroll
  for (unsigned i = 0u; i < 3u; ++i) {
    if (blk[i] < 0)
      return g;
    const unsigned b = (unsigned)blk[i], nj = S::LX * S::XU * (b + 1u) / S::YU;
    if (l < S::LX * nj) {
      g.X0 = S::LX * S::XU * b;
      g.lx = l % S::LX;
      g.y0 = l / S::LX;
      g.dy = nj;
      g.on = true;
      return g;
    }
    l -= S::LX * nj;
  }
  return g;
}

// a lane's chains
template <unsigned NSPLIT> struct GramAcc {
  using S = GramShape<NSPLIT>;
  double a[S::XU][S::YU];
  __device__ __forceinline__ void clear()
  {
#pragma unroll
    for (unsigned u = 0u; u < S::XU; ++u)
#pragma unroll
      for (unsigned v = 0u; v < S::YU; ++v)
        a[u][v] = +0.0;
  }
  __device__ __forceinline__ void tile(const double *const st, const GramLane &g)
  {
    gram_tile<S::XU, S::YU, S::LX>(st, g.X0, g.lx, g.y0, g.dy, a);
  }
  // the entries of the lower triangle: put(offset y * 32 + x, value)
  template <typename F> __device__ __forceinline__ void put(const GramLane &g, const F &f) const
  {
    if (!g.on)
      return;
    const unsigned x0 = g.X0 + g.lx * S::XU;
#pragma unroll
    for (unsigned u = 0u; u < S::XU; ++u)
#pragma unroll
      for (unsigned v = 0u; v < S::YU; ++v) {
        const unsigned y = g.y0 + v * g.dy;
        if (x0 + u >= y)
          f(y * 32u + x0 + u, a[u][v]);
      }
  }
};

// ---------------------------------------------------------------------------
// Right-looking Cholesky of the lower triangle held in R, by two warps with the
// trailing matrix in registers: lane x holds row x, warp 0 its columns 0 .. 15,
// warp 1 its columns 16 .. 31, a[j] = A(x, k + j) in round k.  A round scales
// column k (x > k: times rsqrt_rn(A(k,k))), then every trailing entry takes
// A(x,j) = fma(-A(x,k), A(j,k), A(x,j)) and moves one register down, so that a
// round's indices are constants.  Warp 0 takes rounds 0 .. 15, warp 1 follows it
// with its columns (a barrier of the two per round) and takes the rest.  Every
// entry receives the reference's operations in the reference's order
// (share/device_code_common_Cholesky.hpp:58-158); entries above the diagonal
// are computed too and never used.
// The round's serial chain is the pivot: lane k + 1 updates its own diagonal
// entry (its factor is its own), one shuffle hands it to all lanes, and its
// rsqrt_rn runs beside the trailing updates, whose factors A(j,k) come back
// from shared memory (column k of R, where they belong anyway) by broadcast
// loads: 4 cycles each, which is why one warp for all 32 columns took 6.4 us.
// The square roots of the diagonal are taken together at the end.  With a
// column look-ahead over 8 warps and a barrier per column the pivot's chain was
// barrier, loads, update, shuffle, reciprocal root and root: 9.8 us.
// Afterwards R = L^T with zeros below the diagonal.
// ---------------------------------------------------------------------------
// rounds END - LIVE .. END - LIVE + 7 of the columns up to END - 1, LIVE of them
// alive in the first; with FEED each round's column is handed to warp 1
template <unsigned END, unsigned LIVE, bool FEED>
__device__ __forceinline__ void chol_rounds(double *const R, const unsigned x, double (&a)[16], double &rs,
                                            double &diag, const unsigned feed)
{
#pragma unroll 1
  for (unsigned k = END - LIVE; k < END - LIVE + 8u; ++k) {
    const double l = a[0] * rs;
    if (x == k)
      diag = a[0];
    double *const col = R + k * 32u;
    if (x > k)
      col[x] = l;
    // the next pivot (for k = END - 1 the values below are past the last column and unused)
    const double pv = __shfl_sync(0xffffffffu, __fma_rn(-l, l, a[1]), (k + 1u) & 31u);
    bool ok;
    rs = rsqrt_try(pv, ok);
    if (FEED)
      bar_sync(feed, 64u);
    else
      __syncwarp();
#pragma unroll
    for (unsigned j = 1u; j < LIVE; ++j)
      a[j - 1u] = __fma_rn(-l, col[k + j], a[j]);
    if (!(ok && rsqrt_range(pv)) && k + 1u < END)
      rs = rsqrt_rn_full(pv);
  }
}

// by a group of NW warps (thread gt of the group, named barriers bar and bar +
// 8): the group's warps 0 and 1 factor, all transpose
template <unsigned NW>
__device__ __forceinline__ void chol32_grp(double *const R, const unsigned gt, const unsigned bar)
{
  if (gt < 64u) {
    const unsigned x = gt & 31u;
    double a[16], diag = 0.0, rs;
    if (gt < 32u) {
#pragma unroll
      for (unsigned j = 0u; j < 16u; ++j)
        a[j] = E32(R, x, j);
      rs = rsqrt_rn(__shfl_sync(0xffffffffu, a[0], 0));
      __syncwarp();
      chol_rounds<16u, 16u, true>(R, x, a, rs, diag, bar + 8u);
      chol_rounds<16u, 8u, true>(R, x, a, rs, diag, bar + 8u);
      if (x < 16u)
        E32(R, x, x) = __dsqrt_rn(diag);
    }
    else {
#pragma unroll
      for (unsigned j = 0u; j < 16u; ++j)
        a[j] = E32(R, x, 16u + j);
#pragma unroll 1
      for (unsigned k = 0u; k < 16u; ++k) {
        bar_sync(bar + 8u, 64u);
        const double *const col = R + k * 32u;
        const double l = col[x];
#pragma unroll
        for (unsigned j = 0u; j < 16u; ++j)
          a[j] = __fma_rn(-l, col[16u + j], a[j]);
      }
      rs = rsqrt_rn(__shfl_sync(0xffffffffu, a[0], 16));
      __syncwarp();
      chol_rounds<32u, 16u, false>(R, x, a, rs, diag, 0u);
      chol_rounds<32u, 8u, false>(R, x, a, rs, diag, 0u);
      if (x >= 16u)
        E32(R, x, x) = __dsqrt_rn(diag);
    }
  }
  bar_sync(bar, NW * 32u);
  constexpr unsigned NV = 1024u / (NW * 32u);
  double v[NV];
#pragma unroll
  for (unsigned i = 0u; i < NV; ++i) { // element (x = col of R^T, y = row) = (i*NW*32 + gt)
    const unsigned e = i * NW * 32u + gt, xx = e >> 5, yy = e & 31u;
    v[i] = (xx >= yy) ? E32(R, xx, yy) : 0.0;
  }
  bar_sync(bar, NW * 32u);
#pragma unroll
  for (unsigned i = 0u; i < NV; ++i) {
    const unsigned e = i * NW * 32u + gt, xx = e >> 5, yy = e & 31u;
    E32(R, yy, xx) = v[i];
  }
}

// ---------------------------------------------------------------------------
// Inner Jacobi sweep(s) on R (32x32) accumulating V_loc, by a group of NW warps
// (8, 4 or 2; lane x, warp w of the group, named barrier bar).  An inner step
// has 16 disjoint column pairs; LP = 2 NW lanes take one: lane i of them holds
// NR = 32 / LP rows, i + LP g, of both columns of R and V_loc.
//   The three dot products (Dp, Dq, Apq) are summed in the reference's order
//   (share/device_code_common_Kepler.hpp:26-74: row r adds row r^16, then ^8, ^4,
//   ^2, ^1; IEEE addition commutes): the first log2 NR levels are between the
//   lane's own rows, the others butterflies within the LP lanes.  Every lane
//   evaluates its pair's rotation (branch-free, so the pairs of a warp do not
//   diverge) and applies it to its rows.  One barrier per step.
// Every operation is the reference's (share/device_code_nosort.hpp:4-222,
// share/device_code_cdsort.hpp:25-167, share/device_code_cdsort_KISS.hpp).
// What bounds a step (8 warps): the SM executes one shuffle of a warp per cycle,
// 6 per level of the butterfly and warp, and the rotation is a chain of 540
// cycles.  With a row of two pairs per lane (all 32 lanes summing both pairs by
// a reduce-scatter, then trading the two rotations) a warp had 37 shuffles a
// step, here 24 (18 and 12 with 4 and 2 warps, before 36 and 54 and rotations
// passed through shared memory).
// The rows of neighbouring pairs' lanes are taken in another order (g ^ the
// pair's number), which leaves every sum and keeps their loads in different
// banks.
// ---------------------------------------------------------------------------
template <bool SORT, unsigned NW>
__device__ __forceinline__ void inner_sweeps(double *const R, double *const Vl, const uint8_t *const s0,
                                             const unsigned s0steps, const unsigned nswp, const int definite,
                                             const unsigned npos, unsigned *const red, const unsigned x,
                                             const unsigned w, const unsigned bar, unsigned &blk_s, unsigned &blk_b)
{
  constexpr unsigned LP = 2u * NW, NR = 32u / LP;
  blk_s = 0u;
  blk_b = 0u;
  const unsigned sub = x / LP, i = x % LP;   // the pair's number in the warp, the lane's in the pair
  const unsigned pair = w * (32u / LP) + sub; // the pair of the step
  unsigned row[NR];
#pragma unroll
  for (unsigned g = 0u; g < NR; ++g)
    row[g] = i + LP * (g ^ (sub & (16u / LP - 1u)));
  for (unsigned swp = 0u; swp < nswp; ++swp) {
    unsigned ws = 0u, wb = 0u; // lane 0 of each pair: its counts
    for (unsigned step = 0u; step < s0steps; ++step) {
      const unsigned e = *reinterpret_cast<const uint16_t *>(s0 + step * 32u + 2u * pair), p = e & 255u, q = e >> 8;
      double Gp[NR], Gq[NR], Vp[NR], Vq[NR], dp[NR], dq[NR], pq[NR];
#pragma unroll
      for (unsigned g = 0u; g < NR; ++g) {
        Gp[g] = E32(R, row[g], p);
        Gq[g] = E32(R, row[g], q);
      }
#pragma unroll
      for (unsigned g = 0u; g < NR; ++g) { // loaded now so that the application waits for no load
        Vp[g] = E32(Vl, row[g], p);
        Vq[g] = E32(Vl, row[g], q);
      }
#pragma unroll
      for (unsigned g = 0u; g < NR; ++g) {
        dp[g] = __fma_rn(Gp[g], Gp[g], 0.0);
        dq[g] = __fma_rn(Gq[g], Gq[g], 0.0);
        pq[g] = __fma_rn(Gp[g], Gq[g], 0.0);
      }
#pragma unroll
      for (unsigned k = NR / 2u; k; k >>= 1u)
#pragma unroll
        for (unsigned g = 0u; g < k; ++g) {
          dp[g] = dp[g] + dp[g + k];
          dq[g] = dq[g] + dq[g + k];
          pq[g] = pq[g] + pq[g + k];
        }
#pragma unroll
      for (unsigned k = LP / 2u; k; k >>= 1u) {
        const double a = __shfl_xor_sync(0xffffffffu, dp[0], k), b = __shfl_xor_sync(0xffffffffu, dq[0], k),
                     c = __shfl_xor_sync(0xffffffffu, pq[0], k);
        dp[0] = dp[0] + a;
        dq[0] = dq[0] + b;
        pq[0] = pq[0] + c;
      }
      unsigned a_s, a_b;
      const Rot r = inner_rot<SORT>(dp[0], dq[0], pq[0], p, q, definite, npos, a_s, a_b);
      if (i == 0u) {
        ws += a_s;
        wb += a_b;
      }
      // c = 1 multiplies exactly; a swap of the columns (mode 2) keeps the
      // values; mode 0 leaves them
      if (__any_sync(0xffffffffu, r.mode != 0)) {
        const bool raw = SORT && r.mode == 2;
        const unsigned to_p = (SORT && (raw || r.swap)) ? q : p, to_q = (SORT && (raw || r.swap)) ? p : q;
#pragma unroll
        for (unsigned g = 0u; g < NR; ++g) {
          const double np = r.c * __fma_rn(r.t_, Gq[g], Gp[g]), nq = r.c * __fma_rn(r.t, Gp[g], Gq[g]);
          if (r.mode != 0) {
            E32(R, row[g], to_p) = raw ? Gp[g] : np;
            E32(R, row[g], to_q) = raw ? Gq[g] : nq;
          }
        }
#pragma unroll
        for (unsigned g = 0u; g < NR; ++g) {
          const double np = r.c * __fma_rn(r.t_, Vq[g], Vp[g]), nq = r.c * __fma_rn(r.t, Vp[g], Vq[g]);
          if (r.mode != 0) {
            E32(Vl, row[g], to_p) = raw ? Vp[g] : np;
            E32(Vl, row[g], to_q) = raw ? Vq[g] : nq;
          }
        }
      }
      bar_sync(bar, NW * 32u);
    }
    ws = __reduce_add_sync(0xffffffffu, ws);
    wb = __reduce_add_sync(0xffffffffu, wb);
    if (x == 0u) {
      red[2u * w] = ws;
      red[2u * w + 1u] = wb;
    }
    bar_sync(bar, NW * 32u);
    unsigned tot_s = 0u, tot_b = 0u;
#pragma unroll
    for (unsigned k = 0u; k < NW; ++k) {
      tot_s += red[2u * k];
      tot_b += red[2u * k + 1u];
    }
    bar_sync(bar, NW * 32u);
    if (tot_s) {
      blk_s += tot_s;
      blk_b += tot_b;
    }
    else
      break;
  }
}

// ---------------------------------------------------------------------------
// Update of one 256-row stage: warp rg (0..7), lane = sub + 8*cg.  The thread
// owns rows sub*32 + rg*4 + (0..3) and columns cg*8 + (0..7); entry (u, v)
// adds A[r, s] * B[s, c] for s = (x + c + k) mod 32, k = 0..31, x = r mod 32,
// i.e. the anti-diagonal index t = u + v + k reads column s = x0 + c0 + t.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void update_stage(const double *const st, const double *const VT, const unsigned rg,
                                             const unsigned sub, const unsigned cg, double (&acc)[4][8])
{
  const unsigned x0 = rg * 4u, c0 = cg * 8u;
  const double *const ab = st + sub * 34u + x0;
  const double *const bb = VT + c0;
#pragma unroll
  for (unsigned u = 0u; u < 4u; ++u)
#pragma unroll
    for (unsigned v = 0u; v < 8u; ++v)
      acc[u][v] = +0.0;
#pragma unroll
  for (unsigned t = 0u; t < 42u; ++t) {
    const unsigned s = (x0 + c0 + t) & 31u;
    const double2 a01 = *reinterpret_cast<const double2 *>(ab + s * kUpdColLd);
    const double2 a23 = *reinterpret_cast<const double2 *>(ab + s * kUpdColLd + 2u);
    const double a[4] = {a01.x, a01.y, a23.x, a23.y};
    const double2 b01 = *reinterpret_cast<const double2 *>(bb + s * kVTLd);
    const double2 b23 = *reinterpret_cast<const double2 *>(bb + s * kVTLd + 2u);
    const double2 b45 = *reinterpret_cast<const double2 *>(bb + s * kVTLd + 4u);
    const double2 b67 = *reinterpret_cast<const double2 *>(bb + s * kVTLd + 6u);
    const double b[8] = {b01.x, b01.y, b23.x, b23.y, b45.x, b45.y, b67.x, b67.y};
#pragma unroll
    for (unsigned u = 0u; u < 4u; ++u)
#pragma unroll
      for (unsigned v = 0u; v < 8u; ++v) {
        if ((t >= u + v) && (t - u - v < 32u))
          acc[u][v] = __fma_rn(a[u], b[v], acc[u][v]);
      }
  }
}

// the stage's results in place of its operands: the thread's 4 rows x 8
// columns go where update_stage read them; warp rg read only its own rows
// (rg*4 .. rg*4+3 of each 32-row piece), so after __syncwarp nothing that
// another lane still needs is overwritten.  A TMA store then writes the stage
// back (rows 32-33 of a piece lie outside the view and are not written).
__device__ __forceinline__ void update_put(double *const st, const double (&acc)[4][8], const unsigned rg,
                                           const unsigned sub, const unsigned cg8)
{
  double *const o = st + sub * 34u + rg * 4u;
#pragma unroll
  for (unsigned v = 0u; v < 8u; ++v) {
    double *const col = o + (cg8 * 8u + v) * kUpdColLd;
    *reinterpret_cast<double2 *>(col) = make_double2(acc[0][v], acc[1][v]);
    *reinterpret_cast<double2 *>(col + 2u) = make_double2(acc[2][v], acc[3][v]);
  }
}

// the signature of block pair (iBlk, jBlk): global if the matrix is definite,
// else block-local (share/device_code_nosort_solveV.hpp:33-67)
__device__ __forceinline__ void block_signature(const StepParams &P, const unsigned iBlk, const unsigned jBlk,
                                                int &definite, unsigned &npos)
{
  const unsigned ifc0 = iBlk * kNColB, ifc1 = jBlk * kNColB, nplus = P.nplus;
  if (P.gdefinite) {
    definite = P.gdefinite;
    npos = 0u;
  }
  else if (nplus <= ifc0) {
    npos = 0u;
    definite = -1;
  }
  else if (nplus <= ifc0 + kNColB) {
    npos = nplus - ifc0;
    definite = 0;
  }
  else if (nplus <= ifc1) {
    npos = kNColB;
    definite = 0;
  }
  else if (nplus <= ifc1 + kNColB) {
    npos = kNColB + (nplus - ifc1);
    definite = 0;
  }
  else {
    npos = 2u * kNColB;
    definite = +1;
  }
}

// a block pair's rotation counts into its matrix's sweep counter: big << 32 |
// small, or the low word alone when no rotation was big, as the reference
__device__ __forceinline__ void add_counts(const StepParams &P, const unsigned blk_s, const unsigned blk_b)
{
  if (!blk_s)
    return;
  if (blk_b)
    atomicAdd(P.cvg, (((unsigned long long)blk_b) << 32) | blk_s);
  else
    atomicAdd(reinterpret_cast<unsigned *>(P.cvg), blk_s);
}

// V_loc of block pair `pair`, transposed as update_stage reads it, and whether
// the pair changes, for l1_update_kernel (R is dead)
template <unsigned THREADS>
__device__ __forceinline__ void put_transform(const StepParams &P, const unsigned pair, const bool changes,
                                              double *const R, const double *const Vl)
{
  const unsigned tid = threadIdx.x;
  for (unsigned i = tid; i < 1024u; i += THREADS) {
    const unsigned c = i >> 5, s = i & 31u;
    R[s * kVTLd + c] = E32(Vl, s, c);
  }
  fence_async_shared();
  __syncthreads();
  if (tid == 0u) {
    bulk_s2g(P.vt + (size_t)pair * kTransform, R, kTransform * 8u);
    bulk_commit();
    P.vflag[pair] = changes ? 1u : 0u;
    bulk_wait_all();
  }
}

// ---------------------------------------------------------------------------
// The block-pair step kernel.
// ---------------------------------------------------------------------------
// NBUF update buffers: 2 in the region of the Gram stages, a third (NBUF = 3)
// at kOffUpd3 where the launch provides it
template <bool SORT, bool ACCV, unsigned NSPLIT, unsigned NBUF = 2u, unsigned FAC = 0u>
__device__ __forceinline__ void pair_step(const StepParams &P, const unsigned step, const unsigned pair,
                                          const unsigned rank, double *const sm)
{
  static_assert(FAC == 0u || NSPLIT == 1u, "the QR factor is one CTA's");
  static_assert(NBUF == 2u || NBUF == 3u, "2 or 3 update buffers");
  double *const stg = sm;
  double *const R = sm + kOffR;
  double *const Vl = sm + kOffVl;
  uint8_t *const s0 = reinterpret_cast<uint8_t *>(sm + kOffS0);
  unsigned *const red = reinterpret_cast<unsigned *>(sm + kOffRed);
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kOffBar);

  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const size_t pidx = ((size_t)step * P.pairs + pair) * 2u;
  const unsigned iBlk = P.strat1[pidx + 0u], jBlk = P.strat1[pidx + 1u];

  for (unsigned i = tid; i < 256u; i += kThreads)
    reinterpret_cast<uint32_t *>(s0)[i] = reinterpret_cast<const uint32_t *>(P.strat0)[i];
  if (tid == 0u)
    init_bars(bars);
  __syncthreads();
  if (NSPLIT > 1u)
    cluster_started();
  pdl_wait(); // G, V and the counters are the launch before's

  int failed = 0;
  if constexpr (FAC != 0u) {
    // ----------------- 1'. QR factor (the -DUSE_QR builds) -----------------
    qr_factor_cta(P.G + (size_t)iBlk * kNColB * P.ldG, P.G + (size_t)jBlk * kNColB * P.ldG, P.ldG, P.nrow, R, stg);
  }
  else {
  // ------------------------------ 1. Gram --------------------------------
  const unsigned ntile = P.nrow >> 6; // 64-row tiles
  const GramLane gl = gram_lane<NSPLIT>(rank, warp, lane);
  GramAcc<NSPLIT> gacc;
  gacc.clear();

  const unsigned ngst = (ntile + kGramTiles - 1u) / kGramTiles; // stages of 2 tiles
  // thread 0: the TMA engine brings stage k, per tile block i's and block j's
  // 16 columns as one box each
  auto issue_gram = [&](const unsigned k) {
    const unsigned s = k % kGramStages;
    const unsigned nt = min(kGramTiles, ntile - k * kGramTiles);
    double *const st = stg + s * kGramStage;
    mbar_arrive_expect_tx(&bars[s], nt * 2u * kGramBoxBytes);
    for (unsigned t = 0u; t < nt; ++t) {
      const int tile = (int)(k * kGramTiles + t);
      tma_load_3d(st + t * kGramTileLd, &P.tmGram, 0, tile, (int)(iBlk * kNColB), &bars[s]);
      tma_load_3d(st + t * kGramTileLd + 16u * kGramColLd, &P.tmGram, 0, tile, (int)(jBlk * kNColB), &bars[s]);
    }
  };

  // The Gram warps do not wait for one another: each waits for a stage to land,
  // adds its tiles and arrives on the stage's read barrier; the issuer refills a
  // stage when all have.  (With a CTA barrier per stage of two tiles the phase
  // took 570 cycles a stage more than the tiles do.)
  if (tid == kIssuer) {
    for (unsigned k = 0u; k < ngst; ++k) {
      if (k >= kGramStages &&
          !mbar_wait_bounded(&bars[11u + k % kGramStages], (k / kGramStages - 1u) & 1u, kWaitLimit)) {
        failed = 1;
        break;
      }
      issue_gram(k);
    }
  }
  else if (warp < kGramWarps) {
    for (unsigned k = 0u; k < ngst; ++k) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[k % kGramStages], (k / kGramStages) & 1u, kWaitLimit))) {
        failed = 1;
        break;
      }
      if (gl.on) {
        const unsigned nt = min(kGramTiles, ntile - k * kGramTiles);
        for (unsigned t = 0u; t < nt; ++t)
          gacc.tile(stg + (k % kGramStages) * kGramStage + t * kGramTileLd, gl);
      }
      __syncwarp();
      if (lane == 0u)
        mbar_arrive(&bars[11u + k % kGramStages]);
    }
  }
  failed = __syncthreads_or(failed); // uniform decision
  if (failed && tid == 0u) { // let the copies in flight land (bounded) before anything else, report
    for (unsigned s = 0u; s < kGramStages; ++s)
      for (unsigned par = 0u; par < 2u; ++par)
        (void)mbar_wait_bounded(&bars[s], par, kWaitLimit / 8);
    atomicOr(P.err, kErrWaitTimeout);
  }
  // our share of the lower triangle, into our R and the other CTAs' R
  if (NSPLIT > 1u)
    cluster_wait_started();
  {
    cg::cluster_group cl = cg::this_cluster();
    gacc.put(gl, [&](const unsigned o, const double v) {
      R[o] = v;
#pragma unroll
      for (unsigned q = 1u; q < NSPLIT; ++q)
        cl.map_shared_rank(R, (rank + q) % NSPLIT)[o] = v;
    });
  }
  }
  if (NSPLIT > 1u)
    cg::this_cluster().sync(); // release our writes, acquire the others'
  else
    __syncthreads();
  if (failed)
    return; // the error word is set; the host reports it

  // the first update stage of this CTA: its rows do not change before the
  // update, so the copy overlaps the Cholesky and the inner sweeps
  const unsigned nG = (P.nrow + kUpdRows - 1u) / kUpdRows;
  const unsigned nV = ACCV ? (P.ncol + kUpdRows - 1u) / kUpdRows : 0u;
  const unsigned nst = nG + nV;
  const unsigned nmine = (nst > rank) ? (nst - rank + NSPLIT - 1u) / NSPLIT : 0u;
  auto ubuf = [&](const unsigned s) { return (NBUF == 3u && s == 2u) ? sm + kOffUpd3 : stg + s * kUpdStage; };
  auto issue_upd = [&](const unsigned i) { // one thread: this CTA's i-th stage, 2 tensor copies
    const unsigned k = rank + i * NSPLIT, s = i % NBUF;
    const bool isG = k < nG;
    const CUtensorMap *const tm = isG ? &P.tmG : &P.tmV;
    const int piece = (int)(((isG ? k : (k - nG)) * kUpdRows) >> 5);
    double *const st = ubuf(s);
    mbar_arrive_expect_tx(&bars[4u + s], 2u * kUpdBoxBytes);
    tma_load_3d(st, tm, 0, piece, (int)(iBlk * kNColB), &bars[4u + s]);
    tma_load_3d(st + 16u * kUpdColLd, tm, 0, piece, (int)(jBlk * kNColB), &bars[4u + s]);
  };
  const bool apart = P.vt != nullptr; // the update is another kernel's (l1_update_kernel)
  if (tid == 0u && nmine > 0u && !apart)
    issue_upd(0u);

  // ---------------------------- 2. Cholesky -------------------------------
  for (unsigned i = tid; i < 1024u; i += kThreads)
    Vl[i] = ((i >> 5) == (i & 31u)) ? 1.0 : 0.0;
  if constexpr (FAC == 0u)
    chol32_grp<8u>(R, tid, 0u);
  __syncthreads();

  // --------------------------- 3. inner sweeps ----------------------------
  int definite;
  unsigned npos;
  block_signature(P, iBlk, jBlk, definite, npos);
  unsigned blk_s, blk_b;
  if (FAC == 2u && SORT && definite) // -DUSE_DRMAC: Drmac's sweep in the definite sorting kernels
    drmac_sweeps(R, Vl, s0, P.s0steps, P.nswp0, definite, red, lane, warp, blk_s, blk_b);
  else
    inner_sweeps<SORT, 8u>(R, Vl, s0, P.s0steps, P.nswp0, definite, npos, red, lane, warp, 0u, blk_s, blk_b);

  if (rank == 0u && tid == 0u)
    add_counts(P, blk_s, blk_b);
  if (apart) {
    if (rank == 0u)
      put_transform<kThreads>(P, pair, SORT || blk_s, R, Vl);
    return;
  }
  if (!SORT && !blk_s) { // no rotation: the block pair is unchanged
    if (tid == 0u && nmine > 0u && !mbar_wait_bounded(&bars[4u], 0u, kWaitLimit))
      atomicOr(P.err, kErrWaitTimeout); // the prefetched copy has landed before we leave
    return;
  }

  // ------------------------------ 4. update -------------------------------
  double *const VT = R; // R is dead; B^T[s][c] = V_loc[s][c]
  for (unsigned i = tid; i < 1024u; i += kThreads) {
    const unsigned c = i >> 5, s = i & 31u;
    VT[s * kVTLd + c] = E32(Vl, s, c);
  }

  // The warps do not wait for one another: a warp waits for stage i to land,
  // computes it, puts its results in place (of operands that only it read) and
  // arrives on the stage's done barrier.  Thread 0, before its own stage i, waits
  // for stage i - 1 to be done, stores it with two tensor copies, and issues the
  // copy of stage i + 1 once the store that last used that buffer has read it
  // out (with 3 buffers that of stage i - 2, with 2 that of i - 1, issued just
  // before).  So one warp's stores and barrier latencies overlap the other's
  // arithmetic on its sub-partition (with a CTA barrier per stage they coincided).
  const unsigned rg = warp, sub = lane & 7u, cg8 = lane >> 3;
  auto store_upd = [&](const unsigned i) { // one thread: this CTA's i-th stage back
    const unsigned k = rank + i * NSPLIT;
    const bool isG = k < nG;
    const CUtensorMap *const tm = isG ? &P.tmG : &P.tmV;
    const int piece = (int)(((isG ? k : (k - nG)) * kUpdRows) >> 5);
    double *const sb = ubuf(i % NBUF);
    tma_store_3d(tm, sb, 0, piece, (int)(iBlk * kNColB));
    tma_store_3d(tm, sb + 16u * kUpdColLd, 0, piece, (int)(jBlk * kNColB));
    bulk_commit();
  };
  auto wait_done = [&](const unsigned i) {
    return mbar_wait_bounded(&bars[8u + (i % NBUF)], (i / NBUF) & 1u, kWaitLimit);
  };
  volatile unsigned *const stop = red + 16u; // a wait gave up: all warps leave
  if (tid == 0u)
    *stop = 0u;
  __syncthreads();
  unsigned issued = (nmine > 0u) ? 1u : 0u; // thread 0: copies issued
  int fail = 0;
  for (unsigned i = 0u; i < nmine; ++i) {
    if (tid == 0u) {
      if (i > 0u) {
        if (wait_done(i - 1u))
          store_upd(i - 1u);
        else
          fail = 1;
      }
      if (i + 1u < nmine && !fail) {
        if (NBUF == 3u)
          bulk_wait_read_but1();
        else
          bulk_wait_read();
        issue_upd(i + 1u);
        issued = i + 2u;
      }
    }
    // a warp computes only if all its lanes saw the stage land
    fail = !__all_sync(0xffffffffu, !fail && !*stop &&
                                        mbar_wait_bounded(&bars[4u + (i % NBUF)], (i / NBUF) & 1u, kWaitLimit));
    if (fail) {
      *stop = 1u;
      break;
    }
    double *const sb = ubuf(i % NBUF);
    double acc[4][8]; // the whole warp computes (rows past the end: not stored)
    update_stage(sb, VT, rg, sub, cg8, acc);
    __syncwarp();
    update_put(sb, acc, rg, sub, cg8);
    fence_async_shared();
    __syncwarp();
    if (lane == 0u)
      mbar_arrive(&bars[8u + (i % NBUF)]);
  }
  if (tid == 0u && nmine > 0u && !fail) {
    if (wait_done(nmine - 1u))
      store_upd(nmine - 1u);
    else
      fail = 1;
  }
  fail = __syncthreads_or(fail);
  if (tid == 0u) {
    if (fail) { // the copies in flight land (bounded); report
      for (unsigned q = (issued > 2u) ? issued - 2u : 0u; q < issued; ++q)
        (void)mbar_wait_bounded(&bars[4u + (q % NBUF)], (q / NBUF) & 1u, kWaitLimit / 8);
      atomicOr(P.err, kErrWaitTimeout);
    }
    bulk_wait_all(); // the stores are complete before the block pair counts as done
  }
}

// ---------------------------------------------------------------------------
// Two block pairs in one CTA (batched form; pair A of matrix PA, pair B of
// matrix PB).  The Grams and the updates run on all 8 warps, A's then B's,
// as one stream of stages each (the copies of B's first stages overlap A's
// last ones).  The Cholesky factorisations and the inner sweeps, chains of
// dependent divides and square roots that leave the SM's pipes mostly idle,
// run concurrently: warps 0-3 take pair A (named barrier 1), warps 4-7 pair B
// (barrier 2).  Every entry of R, V_loc and the updated columns is computed
// with the same operations in the same order as by pair_step, so each matrix
// gets the bits it would get alone.
// ---------------------------------------------------------------------------
constexpr unsigned kOffR2 = kSmemDoubles; // pair B's R (later B^T), V_loc, counters
constexpr unsigned kOffVl2 = kOffR2 + 32u * kVTLd;
constexpr unsigned kOffRed2 = kOffVl2 + 1024u;
constexpr unsigned kSmemDoubles2 = kOffRed2 + 16u;

inline size_t batch2_smem_bytes() { return (size_t)kSmemDoubles2 * sizeof(double); }

template <bool SORT, bool ACCV>
__device__ __forceinline__ void pair_step2(const StepParams &PA, const unsigned stepA, const unsigned pairA,
                                           const StepParams &PB, const unsigned stepB, const unsigned pairB,
                                           double *const sm)
{
  double *const stg = sm;
  uint8_t *const s0 = reinterpret_cast<uint8_t *>(sm + kOffS0);
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kOffBar);
  unsigned *const flags = reinterpret_cast<unsigned *>(sm + kOffRed2) + 30u; // [g]: pair g updates

  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  size_t pidx = ((size_t)stepA * PA.pairs + pairA) * 2u;
  const unsigned iA = PA.strat1[pidx + 0u], jA = PA.strat1[pidx + 1u];
  pidx = ((size_t)stepB * PB.pairs + pairB) * 2u;
  const unsigned iB = PB.strat1[pidx + 0u], jB = PB.strat1[pidx + 1u];

  for (unsigned i = tid; i < 256u; i += kThreads)
    reinterpret_cast<uint32_t *>(s0)[i] = reinterpret_cast<const uint32_t *>(PA.strat0)[i];
  if (tid == 0u)
    init_bars(bars);
  __syncthreads();

  pdl_wait();

  // ------------------------------ 1. Grams --------------------------------
  // stages 0 .. ngA-1 are A's, ngA .. ngA+ngB-1 B's
  const unsigned ntA = PA.nrow >> 6, ntB = PB.nrow >> 6;
  const unsigned ngA = (ntA + kGramTiles - 1u) / kGramTiles, ngB = (ntB + kGramTiles - 1u) / kGramTiles;
  const unsigned ng = ngA + ngB;
  const GramLane gl = gram_lane<1u>(0u, warp, lane);
  GramAcc<1u> gacc;
  gacc.clear();
  auto stage_tiles = [&](const unsigned k) {
    return (k < ngA) ? min(kGramTiles, ntA - k * kGramTiles) : min(kGramTiles, ntB - (k - ngA) * kGramTiles);
  };
  auto issue_gram = [&](const unsigned k) {
    const unsigned s = k % kGramStages;
    const bool a = k < ngA;
    const unsigned t0 = (a ? k : (k - ngA)) * kGramTiles, nt = stage_tiles(k);
    const CUtensorMap *const tm = a ? &PA.tmGram : &PB.tmGram;
    const int ci = (int)((a ? iA : iB) * kNColB), cj = (int)((a ? jA : jB) * kNColB);
    double *const st = stg + s * kGramStage;
    mbar_arrive_expect_tx(&bars[s], nt * 2u * kGramBoxBytes);
    for (unsigned t = 0u; t < nt; ++t) {
      tma_load_3d(st + t * kGramTileLd, tm, 0, (int)(t0 + t), ci, &bars[s]);
      tma_load_3d(st + t * kGramTileLd + 16u * kGramColLd, tm, 0, (int)(t0 + t), cj, &bars[s]);
    }
  };
  auto put_gram = [&](double *const R) { // the lower triangle
    gacc.put(gl, [&](const unsigned o, const double v) { R[o] = v; });
    gacc.clear();
  };

  if (tid == kIssuer)
    for (unsigned k = 0u; k + 1u < kGramStages && k < ng; ++k)
      issue_gram(k);
  unsigned k = 0u;
  int failed = 0;
  for (; k < ng; ++k) {
    if (tid == kIssuer && k + kGramStages - 1u < ng)
      issue_gram(k + kGramStages - 1u);
    int fail = 0;
    if (warp < GramShape<1u>::warps) {
      if (!mbar_wait_bounded(&bars[k % kGramStages], (k / kGramStages) & 1u, kWaitLimit))
        fail = 1;
      else if (gl.on) {
        const unsigned nt = stage_tiles(k);
        for (unsigned t = 0u; t < nt; ++t)
          gacc.tile(stg + (k % kGramStages) * kGramStage + t * kGramTileLd, gl);
      }
      if (k + 1u == ngA)
        put_gram(sm + kOffR);
      else if (k + 1u == ng)
        put_gram(sm + kOffR2);
    }
    failed = __syncthreads_or(fail);
    if (failed)
      break;
  }
  if (failed) {
    if (tid == 0u) {
      for (unsigned q = k; q < ng && q < k + kGramStages; ++q)
        (void)mbar_wait_bounded(&bars[q % kGramStages], (q / kGramStages) & 1u, kWaitLimit / 8);
      atomicOr(PA.err, kErrWaitTimeout);
      atomicOr(PB.err, kErrWaitTimeout);
    }
    return;
  }

  // A's first update stage, in flight during the serial phases
  const unsigned nGA = (PA.nrow + kUpdRows - 1u) / kUpdRows, nGB = (PB.nrow + kUpdRows - 1u) / kUpdRows;
  const unsigned nstA = nGA + (ACCV ? (PA.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  const unsigned nstB = nGB + (ACCV ? (PB.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  // update stage geometry: pair g's i-th stage
  auto stage_geom = [&](const unsigned g, const unsigned i, double *&ci, double *&cj, size_t &ld, unsigned &base,
                        unsigned &rows, const CUtensorMap *&tm, int &piece) {
    const StepParams &P = g ? PB : PA;
    const unsigned nG = g ? nGB : nGA, iBlk = g ? iB : iA, jBlk = g ? jB : jA;
    if (i < nG) {
      ci = P.G + (size_t)iBlk * kNColB * P.ldG;
      cj = P.G + (size_t)jBlk * kNColB * P.ldG;
      ld = P.ldG;
      base = i * kUpdRows;
      rows = min(kUpdRows, P.nrow - base);
      tm = &P.tmG;
    }
    else {
      ci = P.V + (size_t)iBlk * kNColB * P.ldV;
      cj = P.V + (size_t)jBlk * kNColB * P.ldV;
      ld = P.ldV;
      base = (i - nG) * kUpdRows;
      rows = min(kUpdRows, P.ncol - base);
      tm = &P.tmV;
    }
    piece = (int)(base >> 5);
  };
  auto issue_upd = [&](const unsigned q, const unsigned g, const unsigned i) { // stream position q
    double *ci, *cj;
    size_t ld;
    unsigned base, rows;
    const CUtensorMap *tm;
    int piece;
    stage_geom(g, i, ci, cj, ld, base, rows, tm, piece);
    const unsigned s = q % kUpdStages;
    double *const st = stg + s * kUpdStage;
    mbar_arrive_expect_tx(&bars[4u + s], 2u * kUpdBoxBytes);
    tma_load_3d(st, tm, 0, piece, (int)((g ? iB : iA) * kNColB), &bars[4u + s]);
    tma_load_3d(st + 16u * kUpdColLd, tm, 0, piece, (int)((g ? jB : jA) * kNColB), &bars[4u + s]);
  };
  if (tid == 0u)
    issue_upd(0u, 0u, 0u);

  // ------------------- 2.-3. Cholesky and inner sweeps --------------------
  {
    const unsigned grp = warp >> 2, gt = tid & 127u, gw = warp & 3u;
    const StepParams &P = grp ? PB : PA;
    double *const R = sm + (grp ? kOffR2 : kOffR);
    double *const Vl = sm + (grp ? kOffVl2 : kOffVl);
    unsigned *const red = reinterpret_cast<unsigned *>(sm + (grp ? kOffRed2 : kOffRed));
    for (unsigned i = gt; i < 1024u; i += 128u)
      Vl[i] = ((i >> 5) == (i & 31u)) ? 1.0 : 0.0;
    chol32_grp<4u>(R, gt, 1u + grp);
    bar_sync(1u + grp, 128u);
    int definite;
    unsigned npos;
    block_signature(P, grp ? iB : iA, grp ? jB : jA, definite, npos);
    unsigned blk_s, blk_b;
    inner_sweeps<SORT, 4u>(R, Vl, s0, P.s0steps, P.nswp0, definite, npos, red, lane, gw, 1u + grp, blk_s, blk_b);
    if (gt == 0u) {
      add_counts(P, blk_s, blk_b);
      flags[grp] = (SORT || blk_s) ? 1u : 0u;
    }
  }
  __syncthreads();
  const bool updA = flags[0] != 0u, updB = flags[1] != 0u;
  // the stream of update stages: A's (or, when A is unchanged, its prefetched
  // first stage, waited for and dropped), then B's
  const unsigned qa = updA ? nstA : 1u, nq = qa + (updB ? nstB : 0u);
  if (nq == 1u && !updA) {
    if (tid == 0u && !mbar_wait_bounded(&bars[4u], 0u, kWaitLimit))
      atomicOr(PA.err, kErrWaitTimeout);
    return;
  }

  // ------------------------------ 4. updates ------------------------------
  for (unsigned i = tid; i < 2048u; i += kThreads) { // both R are dead: B^T[s][c] = V_loc[s][c]
    const unsigned g = i >> 10, c = (i >> 5) & 31u, s_ = i & 31u;
    (sm + (g ? kOffR2 : kOffR))[s_ * kVTLd + c] = E32(sm + (g ? kOffVl2 : kOffVl), s_, c);
  }
  __syncthreads();
  const unsigned rg = warp, sub = lane & 7u, cg8 = lane >> 3;
  for (unsigned q = 0u; q < nq; ++q) {
    if (tid == 0u && q + 1u < nq) {
      const unsigned q1 = q + 1u;
      bulk_wait_read(); // the store of stage q - 1 has read the buffer stage q + 1 lands in
      if (q1 < qa)
        issue_upd(q1, 0u, q1);
      else
        issue_upd(q1, 1u, q1 - qa);
    }
    const int fail = !__all_sync(0xffffffffu, mbar_wait_bounded(&bars[4u + (q % kUpdStages)], (q / kUpdStages) & 1u,
                                                                kWaitLimit));
    const unsigned g = (q < qa) ? 0u : 1u;
    const bool work = g == 1u || updA;
    double *const sb = stg + (q % kUpdStages) * kUpdStage;
    if (!fail && work) {
      double acc[4][8];
      update_stage(sb, sm + (g ? kOffR2 : kOffR), rg, sub, cg8, acc);
      __syncwarp();
      update_put(sb, acc, rg, sub, cg8);
      fence_async_shared();
    }
    if (__syncthreads_or(fail)) {
      if (tid == 0u) {
        (void)mbar_wait_bounded(&bars[4u + (q % kUpdStages)], (q / kUpdStages) & 1u, kWaitLimit / 8);
        if (q + 1u < nq)
          (void)mbar_wait_bounded(&bars[4u + ((q + 1u) % kUpdStages)], ((q + 1u) / kUpdStages) & 1u,
                                  kWaitLimit / 8);
        bulk_wait_all();
        atomicOr(g ? PB.err : PA.err, kErrWaitTimeout);
      }
      return;
    }
    if (tid == 0u && work) {
      double *ci, *cj;
      size_t ld;
      unsigned base, rows;
      const CUtensorMap *tm;
      int piece;
      stage_geom(g, g ? q - qa : q, ci, cj, ld, base, rows, tm, piece);
      tma_store_3d(tm, sb, 0, piece, (int)((g ? iB : iA) * kNColB));
      tma_store_3d(tm, sb + 16u * kUpdColLd, 0, piece, (int)((g ? jB : jA) * kNColB));
      bulk_commit();
    }
  }
  if (tid == 0u)
    bulk_wait_all();
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ---------------------------------------------------------------------------
// One block pair on a CTA of 4 warps (batched form, two such CTAs per SM).
// The arithmetic is that of pair_step with one CTA per pair -- the Gram
// chains of pair_step with one CTA per pair on warps 0-2 (warp 3 issues the tile copies), the
// Cholesky factorisation and inner sweeps of pair_step2's warp
// groups, pair_step's update tiles (warp w takes row groups w and w + 4 of
// every stage) -- so every matrix gets the bits of its single call.  Shared
// memory (86 KB): the Gram's 4 stages of one 64-row tile, later one update
// buffer; R, V_loc.  With one buffer a stage's copy waits for the store of
// the stage before; the other CTA of the SM runs meanwhile, and its serial
// phases (Cholesky, inner sweeps: chains of divides and square roots that
// leave the pipes idle) overlap this CTA's Gram and update, and the reverse.
// ---------------------------------------------------------------------------
constexpr unsigned kNThreads = 128u;
constexpr unsigned kNGStages = 4u;
constexpr unsigned kNIssuer = 96u; // lane 0 of warp 3
constexpr unsigned kNRegion = (kNGStages * kGramTileLd > kUpdStage) ? kNGStages * kGramTileLd : kUpdStage;
constexpr unsigned kNOffR = kNRegion; // R, 32x32 (later B^T, 32x34)
constexpr unsigned kNOffVl = kNOffR + 32u * kVTLd;
constexpr unsigned kNOffS0 = kNOffVl + 1024u;
constexpr unsigned kNOffRed = kNOffS0 + 128u;
constexpr unsigned kNOffBar = kNOffRed + 16u; // [0..3] Gram stages, [4] the update buffer, [5..8] Gram stages read
constexpr unsigned kNBars = 9u;
constexpr unsigned kNSmemDoubles = kNOffBar + 10u;
static_assert(2u * (kNSmemDoubles * sizeof(double) + 1024u) <= 228u * 1024u, "two CTAs per SM");
inline size_t batchn_smem_bytes() { return (size_t)kNSmemDoubles * sizeof(double); }

__device__ __forceinline__ void init_bars_n(uint64_t *const bars)
{
  for (unsigned b = 0u; b < kNBars; ++b)
    mbar_init(&bars[b], (b < 5u) ? 1u : kGramWarps);
  mbar_fence_init();
}

__device__ __forceinline__ void inval_bars_n(uint64_t *const bars)
{
  for (unsigned b = 0u; b < kNBars; ++b)
    mbar_inval(&bars[b]);
}

// The Gram phase of a CTA of 4 warps over nt tiles, one per stage: issue(k) by a
// lane of warp 3 into stage k mod 4 once the Gram warps have read tile k - 4,
// add(k) by each Gram warp when tile k has landed.  1 if a wait gave up.
template <typename I, typename A>
__device__ __forceinline__ int gram_phase_n(uint64_t *const bars, const unsigned nt, const I &issue, const A &add)
{
  const unsigned tid = threadIdx.x, warp = tid >> 5;
  int failed = 0;
  if (tid == kNIssuer) {
    for (unsigned k = 0u; k < nt && !failed; ++k) {
      if (k >= kNGStages && !mbar_wait_bounded(&bars[5u + k % kNGStages], (k / kNGStages - 1u) & 1u, kWaitLimit))
        failed = 1;
      else
        issue(k);
    }
  }
  else if (warp < kGramWarps) {
    for (unsigned k = 0u; k < nt && !failed; ++k) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[k % kNGStages], (k / kNGStages) & 1u, kWaitLimit)))
        failed = 1;
      else {
        add(k);
        __syncwarp();
        if ((tid & 31u) == 0u)
          mbar_arrive(&bars[5u + k % kNGStages]);
      }
    }
  }
  failed = __syncthreads_or(failed);
  if (failed && tid == 0u) // the copies in flight land (bounded) before anything else
    for (unsigned b = 0u; b < kNGStages; ++b)
      for (unsigned par = 0u; par < 2u; ++par)
        (void)mbar_wait_bounded(&bars[b], par, kWaitLimit / 8);
  return failed;
}

template <bool SORT, bool ACCV>
__device__ __forceinline__ void pair_step_n(const StepParams &P, const unsigned step, const unsigned pair,
                                            double *const sm)
{
  double *const stg = sm;
  double *const R = sm + kNOffR;
  double *const Vl = sm + kNOffVl;
  uint8_t *const s0 = reinterpret_cast<uint8_t *>(sm + kNOffS0);
  unsigned *const red = reinterpret_cast<unsigned *>(sm + kNOffRed);
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kNOffBar);
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const size_t pidx = ((size_t)step * P.pairs + pair) * 2u;
  const unsigned iBlk = P.strat1[pidx + 0u], jBlk = P.strat1[pidx + 1u];

  for (unsigned i = tid; i < 256u; i += kNThreads)
    reinterpret_cast<uint32_t *>(s0)[i] = reinterpret_cast<const uint32_t *>(P.strat0)[i];
  if (tid == 0u)
    init_bars_n(bars);
  __syncthreads();

  pdl_wait(); // G, V and the counters are the launch before's

  // ------------------------------ 1. Gram --------------------------------
  const unsigned ntile = P.nrow >> 6;
  const GramLane gl = gram_lane<1u>(0u, warp, lane);
  GramAcc<1u> gacc;
  gacc.clear();
  auto issue_gram = [&](const unsigned k) { // tile k into stage k mod 4
    const unsigned s = k % kNGStages;
    double *const st = stg + s * kGramTileLd;
    mbar_arrive_expect_tx(&bars[s], 2u * kGramBoxBytes);
    tma_load_3d(st, &P.tmGram, 0, (int)k, (int)(iBlk * kNColB), &bars[s]);
    tma_load_3d(st + 16u * kGramColLd, &P.tmGram, 0, (int)k, (int)(jBlk * kNColB), &bars[s]);
  };
  if (gram_phase_n(bars, ntile, issue_gram, [&](const unsigned k) {
        if (gl.on)
          gacc.tile(stg + (k % kNGStages) * kGramTileLd, gl);
      })) {
    if (tid == 0u)
      atomicOr(P.err, kErrWaitTimeout);
    return;
  }
  gacc.put(gl, [&](const unsigned o, const double v) { R[o] = v; });
  __syncthreads();

  // the first update stage: its rows do not change before the update, so the
  // copy overlaps the Cholesky and the inner sweeps
  const unsigned nG = (P.nrow + kUpdRows - 1u) / kUpdRows;
  const unsigned nst = nG + (ACCV ? (P.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  auto issue_upd = [&](const unsigned i) {
    const bool isG = i < nG;
    const CUtensorMap *const tm = isG ? &P.tmG : &P.tmV;
    const int piece = (int)(((isG ? i : (i - nG)) * kUpdRows) >> 5);
    mbar_arrive_expect_tx(&bars[4], 2u * kUpdBoxBytes);
    tma_load_3d(stg, tm, 0, piece, (int)(iBlk * kNColB), &bars[4]);
    tma_load_3d(stg + 16u * kUpdColLd, tm, 0, piece, (int)(jBlk * kNColB), &bars[4]);
  };
  const bool apart = P.vt != nullptr; // the update is another kernel's (l1_update_kernel)
  if (tid == 0u && nst > 0u && !apart)
    issue_upd(0u);

  // ------------------- 2.-3. Cholesky and inner sweeps --------------------
  for (unsigned i = tid; i < 1024u; i += kNThreads)
    Vl[i] = ((i >> 5) == (i & 31u)) ? 1.0 : 0.0;
  chol32_grp<4u>(R, tid, 0u);
  __syncthreads();
  int definite;
  unsigned npos;
  block_signature(P, iBlk, jBlk, definite, npos);
  unsigned blk_s, blk_b;
  inner_sweeps<SORT, 4u>(R, Vl, s0, P.s0steps, P.nswp0, definite, npos, red, lane, warp, 0u, blk_s, blk_b);
  if (tid == 0u)
    add_counts(P, blk_s, blk_b);
  if (apart) {
    put_transform<kNThreads>(P, pair, SORT || blk_s, R, Vl);
    return;
  }
  if (!SORT && !blk_s) { // no rotation: the block pair is unchanged
    if (tid == 0u && nst > 0u && !mbar_wait_bounded(&bars[4], 0u, kWaitLimit))
      atomicOr(P.err, kErrWaitTimeout); // the prefetched copy has landed before we leave
    return;
  }

  // ------------------------------ 4. update -------------------------------
  for (unsigned i = tid; i < 1024u; i += kNThreads) { // R is dead: B^T[s][c] = V_loc[s][c]
    const unsigned c = i >> 5, s_ = i & 31u;
    R[s_ * kVTLd + c] = E32(Vl, s_, c);
  }
  __syncthreads();
  const unsigned sub = lane & 7u, cg8 = lane >> 3;
  for (unsigned i = 0u; i < nst; ++i) {
    if (tid == 0u && i > 0u) {
      bulk_wait_read(); // the store of stage i - 1 has read the buffer out
      issue_upd(i);
    }
    const int fail = !__all_sync(0xffffffffu, mbar_wait_bounded(&bars[4], i & 1u, kWaitLimit));
    if (!fail) {
#pragma unroll 1
      for (unsigned h = 0u; h < 2u; ++h) { // row groups warp and warp + 4
        double acc[4][8];
        update_stage(stg, R, warp + 4u * h, sub, cg8, acc);
        __syncwarp();
        update_put(stg, acc, warp + 4u * h, sub, cg8);
      }
      fence_async_shared();
    }
    if (__syncthreads_or(fail)) {
      if (tid == 0u) {
        (void)mbar_wait_bounded(&bars[4], i & 1u, kWaitLimit / 8);
        bulk_wait_all();
        atomicOr(P.err, kErrWaitTimeout);
      }
      return;
    }
    if (tid == 0u) {
      const bool isG = i < nG;
      const CUtensorMap *const tm = isG ? &P.tmG : &P.tmV;
      const int piece = (int)(((isG ? i : (i - nG)) * kUpdRows) >> 5);
      tma_store_3d(tm, stg, 0, piece, (int)(iBlk * kNColB));
      tma_store_3d(tm, stg + 16u * kUpdColLd, 0, piece, (int)(jBlk * kNColB));
      bulk_commit();
    }
  }
  if (tid == 0u)
    bulk_wait_all(); // the stores are complete before the block pair counts as done
}

// ---------------------------------------------------------------------------
// Two block pairs on a CTA of 4 warps (batched form, two such CTAs per SM:
// four pairs in flight per SM).  Pair A of matrix PA, pair B of matrix PB:
// their Grams (warps 0-2, copies by warp 3) and updates (warp w
// takes row groups w and w + 4 of every stage) run on the 4 warps, A's then
// B's, as one stream of tiles and one of stages; their Cholesky
// factorisations and inner sweeps run concurrently, warps 0-1 on A (named
// barrier 1), warps 2-3 on B (barrier 2).
// Every entry gets the operations of pair_step in the
// same order, so each matrix gets the bits of its single call.  Shared
// memory (104 KB): the Gram's 4 stages of one tile, later one update buffer;
// A's and B's R, V_loc and counters.
// ---------------------------------------------------------------------------
constexpr unsigned kN2OffRA = kNRegion;
constexpr unsigned kN2OffVlA = kN2OffRA + 32u * kVTLd;
constexpr unsigned kN2OffRB = kN2OffVlA + 1024u;
constexpr unsigned kN2OffVlB = kN2OffRB + 32u * kVTLd;
constexpr unsigned kN2OffS0 = kN2OffVlB + 1024u;
constexpr unsigned kN2OffRed = kN2OffS0 + 128u; // [0..3] A's counts, [4..7] B's, [8..9] flags
constexpr unsigned kN2OffBar = kN2OffRed + 8u;  // as kNOffBar
constexpr unsigned kN2SmemDoubles = kN2OffBar + 10u;
static_assert(2u * (kN2SmemDoubles * sizeof(double) + 1024u) <= 228u * 1024u, "two CTAs per SM");
inline size_t batchn2_smem_bytes() { return (size_t)kN2SmemDoubles * sizeof(double); }

template <bool SORT, bool ACCV>
__device__ __forceinline__ void pair_step2n(const StepParams &PA, const unsigned stepA, const unsigned pairA,
                                            const StepParams &PB, const unsigned stepB, const unsigned pairB,
                                            double *const sm)
{
  double *const stg = sm;
  uint8_t *const s0 = reinterpret_cast<uint8_t *>(sm + kN2OffS0);
  unsigned *const red = reinterpret_cast<unsigned *>(sm + kN2OffRed);
  uint64_t *const bars = reinterpret_cast<uint64_t *>(sm + kN2OffBar);
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  size_t pidx = ((size_t)stepA * PA.pairs + pairA) * 2u;
  const unsigned iA = PA.strat1[pidx + 0u], jA = PA.strat1[pidx + 1u];
  pidx = ((size_t)stepB * PB.pairs + pairB) * 2u;
  const unsigned iB = PB.strat1[pidx + 0u], jB = PB.strat1[pidx + 1u];

  for (unsigned i = tid; i < 256u; i += kNThreads)
    reinterpret_cast<uint32_t *>(s0)[i] = reinterpret_cast<const uint32_t *>(PA.strat0)[i];
  if (tid == 0u)
    init_bars_n(bars);
  __syncthreads();

  // ------------------------------ 1. Grams --------------------------------
  // tiles 0 .. ntA-1 are A's, ntA .. ntA+ntB-1 B's
  const unsigned ntA = PA.nrow >> 6, ntB = PB.nrow >> 6, nt = ntA + ntB;
  const GramLane gl = gram_lane<1u>(0u, warp, lane);
  GramAcc<1u> gacc;
  gacc.clear();
  auto issue_gram = [&](const unsigned k) {
    const unsigned s = k % kNGStages;
    const bool a = k < ntA;
    const CUtensorMap *const tm = a ? &PA.tmGram : &PB.tmGram;
    const int tile = (int)(a ? k : (k - ntA));
    double *const st = stg + s * kGramTileLd;
    mbar_arrive_expect_tx(&bars[s], 2u * kGramBoxBytes);
    tma_load_3d(st, tm, 0, tile, (int)((a ? iA : iB) * kNColB), &bars[s]);
    tma_load_3d(st + 16u * kGramColLd, tm, 0, tile, (int)((a ? jA : jB) * kNColB), &bars[s]);
  };
  auto put_gram = [&](double *const R) { // the lower triangle
    gacc.put(gl, [&](const unsigned o, const double v) { R[o] = v; });
    gacc.clear();
  };
  if (gram_phase_n(bars, nt, issue_gram, [&](const unsigned k) {
        if (gl.on)
          gacc.tile(stg + (k % kNGStages) * kGramTileLd, gl);
        if (k + 1u == ntA)
          put_gram(sm + kN2OffRA);
        else if (k + 1u == nt)
          put_gram(sm + kN2OffRB);
      })) {
    if (tid == 0u) {
      atomicOr(PA.err, kErrWaitTimeout);
      atomicOr(PB.err, kErrWaitTimeout);
    }
    return;
  }

  // the update stages: A's, then B's; A's first one in flight during the
  // serial phases
  const unsigned nGA = (PA.nrow + kUpdRows - 1u) / kUpdRows, nGB = (PB.nrow + kUpdRows - 1u) / kUpdRows;
  const unsigned nstA = nGA + (ACCV ? (PA.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  const unsigned nstB = nGB + (ACCV ? (PB.ncol + kUpdRows - 1u) / kUpdRows : 0u);
  auto stage_at = [&](const unsigned g, const unsigned i, const CUtensorMap *&tm, int &piece) {
    const StepParams &P = g ? PB : PA;
    const unsigned nG = g ? nGB : nGA;
    const bool isG = i < nG;
    tm = isG ? &P.tmG : &P.tmV;
    piece = (int)(((isG ? i : (i - nG)) * kUpdRows) >> 5);
  };
  auto issue_upd = [&](const unsigned g, const unsigned i) {
    const CUtensorMap *tm;
    int piece;
    stage_at(g, i, tm, piece);
    mbar_arrive_expect_tx(&bars[4], 2u * kUpdBoxBytes);
    tma_load_3d(stg, tm, 0, piece, (int)((g ? iB : iA) * kNColB), &bars[4]);
    tma_load_3d(stg + 16u * kUpdColLd, tm, 0, piece, (int)((g ? jB : jA) * kNColB), &bars[4]);
  };
  if (tid == 0u && nstA > 0u)
    issue_upd(0u, 0u);

  // ------------------- 2.-3. Cholesky and inner sweeps --------------------
  {
    const unsigned grp = warp >> 1, gt = tid & 63u, gw = warp & 1u;
    const StepParams &P = grp ? PB : PA;
    double *const R = sm + (grp ? kN2OffRB : kN2OffRA);
    double *const Vl = sm + (grp ? kN2OffVlB : kN2OffVlA);
    for (unsigned i = gt; i < 1024u; i += 64u)
      Vl[i] = ((i >> 5) == (i & 31u)) ? 1.0 : 0.0;
    chol32_grp<2u>(R, gt, 1u + grp);
    bar_sync(1u + grp, 64u);
    int definite;
    unsigned npos;
    block_signature(P, grp ? iB : iA, grp ? jB : jA, definite, npos);
    unsigned blk_s, blk_b;
    inner_sweeps<SORT, 2u>(R, Vl, s0, P.s0steps, P.nswp0, definite, npos, red + 4u * grp, lane, gw, 1u + grp, blk_s,
                           blk_b);
    if (gt == 0u) {
      add_counts(P, blk_s, blk_b);
      red[8u + grp] = (SORT || blk_s) ? 1u : 0u;
    }
  }
  __syncthreads();
  const bool updA = red[8] != 0u, updB = red[9] != 0u;
  // the stream of update stages: A's (or, when A is unchanged, its prefetched
  // first stage, waited for and dropped), then B's
  const unsigned qa = updA ? nstA : (nstA > 0u ? 1u : 0u), nq = qa + (updB ? nstB : 0u);
  if (nq == qa && !updA) {
    if (tid == 0u && qa > 0u && !mbar_wait_bounded(&bars[4], 0u, kWaitLimit))
      atomicOr(PA.err, kErrWaitTimeout);
    return;
  }

  // ------------------------------ 4. updates ------------------------------
  for (unsigned i = tid; i < 2048u; i += kNThreads) { // both R are dead: B^T[s][c] = V_loc[s][c]
    const unsigned g = i >> 10, c = (i >> 5) & 31u, s_ = i & 31u;
    (sm + (g ? kN2OffRB : kN2OffRA))[s_ * kVTLd + c] = E32(sm + (g ? kN2OffVlB : kN2OffVlA), s_, c);
  }
  __syncthreads();
  const unsigned sub = lane & 7u, cg8 = lane >> 3;
  for (unsigned q = 0u; q < nq; ++q) {
    const unsigned g = (q < qa) ? 0u : 1u, i = g ? q - qa : q;
    if (tid == 0u && q > 0u) {
      bulk_wait_read(); // the store of stage q - 1 has read the buffer out
      issue_upd(g, i);
    }
    const int fail = !__all_sync(0xffffffffu, mbar_wait_bounded(&bars[4], q & 1u, kWaitLimit));
    const bool work = g == 1u || updA;
    if (!fail && work) {
#pragma unroll 1
      for (unsigned h = 0u; h < 2u; ++h) { // row groups warp and warp + 4
        double acc[4][8];
        update_stage(stg, sm + (g ? kN2OffRB : kN2OffRA), warp + 4u * h, sub, cg8, acc);
        __syncwarp();
        update_put(stg, acc, warp + 4u * h, sub, cg8);
      }
      fence_async_shared();
    }
    if (__syncthreads_or(fail)) {
      if (tid == 0u) {
        (void)mbar_wait_bounded(&bars[4], q & 1u, kWaitLimit / 8);
        bulk_wait_all();
        atomicOr(g ? PB.err : PA.err, kErrWaitTimeout);
      }
      return;
    }
    if (tid == 0u && work) {
      const CUtensorMap *tm;
      int piece;
      stage_at(g, i, tm, piece);
      tma_store_3d(tm, stg, 0, piece, (int)((g ? iB : iA) * kNColB));
      tma_store_3d(tm, stg + 16u * kUpdColLd, 0, piece, (int)((g ? jB : jA) * kNColB));
      bulk_commit();
    }
  }
  if (tid == 0u)
    bulk_wait_all();
}

} // namespace gjx
