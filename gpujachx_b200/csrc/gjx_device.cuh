// gjx_device.cuh -- sm_100a device primitives of the blocked one-sided Jacobi.
//
// Every arithmetic routine here produces the same bits as the corresponding
// reference routine (share/device_code_common*.hpp): the operations are IEEE
// correctly rounded (__fma_rn, __ddiv_rn, __dsqrt_rn, __drcp_rn) and are
// applied in the reference's order, so a block-pair step computed here equals
// the reference's bit for bit.  This file is compiled with --fmad=false so
// that no a*b+c is contracted behind our back.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "gjx_internal.h"

namespace gjx {

// sqrt(2^-53), sqrt(2/2^-53) = 2^27, sqrt(32)*2^-53, 2/sqrt(3), 1/2:
// correctly rounded values of the definitions in share/HypJacL.hpp:21-59.
constexpr double kSqrtHeps = 0x1.6a09e667f3bcdp-27;
constexpr double kSqrt2Heps = 0x1.0p+27;
constexpr double kMyTol = 0x1.6a09e667f3bcdp-51;
constexpr double kCoshIFix = 0x1.279a74590331cp+0;
constexpr double kTanh1Fix = 0.5;


// ---------------------------------------------------------------------------
// correctly rounded 1/sqrt
// ---------------------------------------------------------------------------

// Is 1/sqrt(F) above the midpoint (2Y+1) * 2^-80, i.e. (2Y+1)^2 * F < 2^160?
__device__ __forceinline__ bool above_mid(const unsigned long long y2p1, const unsigned long long F)
{
  const unsigned long long Pl = y2p1 * y2p1;             // (2Y+1)^2 < 2^108
  const unsigned long long Ph = __umul64hi(y2p1, y2p1);
  const unsigned long long lo_hi = __umul64hi(Pl, F);    // (Pl * F) >> 64
  const unsigned long long hh_lo = Ph * F;               // Ph * F < 2^98
  const unsigned long long hh_hi = __umul64hi(Ph, F);
  const unsigned long long T_lo = hh_lo + lo_hi;         // (P * F) >> 64
  const unsigned long long T_hi = hh_hi + (T_lo < hh_lo ? 1ull : 0ull);
  return T_hi < (1ull << 32);                            // (P * F) >> 64 < 2^96
}

// 2^k as a double, k in [-1022, 1023]
__device__ __forceinline__ double pow2(const int k) { return __longlong_as_double((long long)(k + 1023) << 52); }

// 1/sqrt(a) rounded to nearest.  Our own method.  Scale a = f * 4^k with
// f in [1, 4), so that 1/sqrt(f) = Y * 2^-53 lies in (1/2, 1) with Y a
// 53-bit integer after rounding.  From rsqrt()'s value y (here in the whole
// method; rsqrt_try below is the usual way):
//   * mostly (after P. Markstein, "IA-64 and Elementary Functions"):
//     e = 1 - f y^2 by two FMAs on y^2 = yh + yl (error below 2^-103), then
//     1/sqrt(f) = y (1 + e/2 + O(e^2)); in ulps the correction is
//     d = 2^53 y e / 2 within 2^-48, so Y = y 2^53 + rint(d) unless d lies
//     within 2^-40 of a half-integer;
//   * otherwise (almost never), the exact test: 1/sqrt(f) lies above the
//     midpoint (2Y+1) * 2^-54 iff (2Y+1)^2 * F < 2^160, F = f 2^52, decided
//     in integers.
// Any correctly rounded 1/sqrt returns these bits.
static __device__ __noinline__ long long rsqrt_fix_exact(long long Y, const unsigned long long F)
{
  for (int i = 0; (i < 4) && above_mid((unsigned long long)(2 * Y + 1), F); ++i)
    ++Y;
  for (int i = 0; (i < 4) && (Y > (1ll << 52)) && !above_mid((unsigned long long)(2 * Y - 1), F); ++i)
    --Y;
  return Y;
}

// the whole method, every input class; the slow path of rsqrt_rn below
static __device__ __noinline__ double rsqrt_rn_full(const double a)
{
  unsigned long long bits = (unsigned long long)__double_as_longlong(a);
  if ((bits >> 63) || ((bits >> 52) == 0x7FFu) || !(bits << 1)) { // negative, inf, nan, zero
    if (isnan(a))
      return a + a;
    if (a == 0.0)
      return copysign(__longlong_as_double(0x7ff0000000000000ll), a);
    if (a < 0.0)
      return __longlong_as_double((long long)0xfff8000000000000ull);
    return 0.0; // +inf
  }
  int sh = 0; // a = a' * 2^-sh with a' normal
  double an = a;
  if (!(bits >> 52)) {
    an = a * pow2(108);
    bits = (unsigned long long)__double_as_longlong(an);
    sh = 108;
  }
  const double ya = rsqrt(an);              // estimate of 1/sqrt(a'), within an ulp
  const int eu = (int)(bits >> 52) - 1023; // a' = m * 2^eu, m in [1, 2)
  const int k2 = eu & ~1;                  // a' = f * 2^k2, f in [1, 4)
  const double f = __longlong_as_double((long long)((bits & 0xFFFFFFFFFFFFFull) | ((unsigned long long)(1023 + (eu - k2)) << 52)));
  const int kk = (k2 - sh) / 2; // a = f * 4^kk exactly (k2 - sh is even)
  if (f == 1.0)
    return pow2(-kk);
  const double y = ya * pow2(k2 / 2); // estimate of 1/sqrt(f), in (1/2, 1] (exact scaling)
  const double yh = y * y;
  const double yl = __fma_rn(y, y, -yh);
  const double e = __fma_rn(-f, yl, __fma_rn(-f, yh, 1.0));
  const double d = (y * (0.5 * e)) * pow2(53);
  const double dr = rint(d);
  double Yd = __fma_rn(y, pow2(53), dr); // y 2^53 + rint(d): an integer below 2^54, exact
  if (fabs(d - dr) > 0.5 - 0x1.0p-40 || Yd >= pow2(53) || Yd < pow2(52)) {
    long long Y = (long long)fmin(fmax(Yd, pow2(52)), pow2(53) - 1.0);
    Yd = (double)rsqrt_fix_exact(Y, (unsigned long long)(f * pow2(52)));
  }
  return Yd * pow2(-53 - kk); // exact scaling into the normal range
}

// ---------------------------------------------------------------------------
// Correctly rounded reciprocal square root, quotient, reciprocal and square
// root without branches.  Each takes the hardware's estimate (rsqrt.approx /
// rcp.approx, relative error about 2^-20, measured), corrects it, and PROVES
// the result; ok is false when the proof fails -- almost never for the
// operands of a rotation, always for zeros, infinities, NaN, subnormals and
// results that are a power of 2 (where the spacing halves below) -- and the
// caller then takes the IEEE operation.  Without branches the chains of a
// rotation overlap, which calls of the IEEE operations (each with a branch to
// its special cases) do not.  The proofs compare high words as integers
// (hi(|x|) < hi(y) implies |x| < y), so they cost the FP64 pipe, which the
// warps of a sub-partition share, one or two operations each.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int hi_abs(const double a) { return __double2hiint(a) & 0x7FFFFFFF; }
__device__ __forceinline__ int hi_binade(const double a) { return __double2hiint(a) & 0x7FF00000; }
__device__ __forceinline__ bool pow2_significand(const double a)
{
  return !((__double2hiint(a) & 0xFFFFF) | __double2loint(a));
}

__device__ __forceinline__ double rsqrt_estimate(const double a)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return __hiloint2double(__double2hiint(y), 0);
}

// The estimate y0 has no low word, so y0^2 is exact and the residual e = 1 -
// a y0^2 takes one FMA; 1/sqrt(a) = y0 (1 - e)^(-1/2) = y0 + (y0 e) (1/2 + 3/8 e
// + 5/16 e^2 + 35/128 e^3), the next term below 2^-90 (|e| < 2^-18 is checked).
// The correction is known to 2^-16 of half an ulp of the result c, so c, its
// sum with y0 rounded once, is 1/sqrt(a) rounded to nearest if it differs from
// the unrounded sum by less than (1 - 2^-15) / 2 ulp (c - y0 is exact).  The
// caller sees to a within 2^+-960, where y0^2 and a y0^2 stay normal.
// A chain of 7 operations: 100 cycles (191 before, with the estimate refined to
// an ulp first).
__device__ __forceinline__ double rsqrt_try(const double a, bool &ok)
{
  const double y0 = rsqrt_estimate(a);
  const double e = __fma_rn(-a, y0 * y0, 1.0);
  const double ye = y0 * e;
  const double w = __fma_rn(e * e, __fma_rn(0.2734375, e, 0.3125), __fma_rn(0.375, e, 0.5));
  const double c = __fma_rn(ye, w, y0);
  const double z = __fma_rn(ye, w, y0 - c);
  ok = (hi_abs(z) < hi_binade(c) - (53 << 20) - 64) && !pow2_significand(c) && (hi_abs(e) < ((1023 - 18) << 20));
  return c;
}

// h / a and 1 / a: the quotient to 2^-40 by one Newton step, then its residual
// (after P. Markstein, "IA-64 and Elementary Functions").  q is the quotient
// rounded to nearest if |h - a q| < |a| ulp(q) / 2; the residual is rounded
// once, which the comparison of high words covers.  The caller sees to
// |h| >= 2^-900 (or zero).
__device__ __forceinline__ bool quotient_ok(const double rho, const double a, const double q)
{
  return (hi_abs(rho) < hi_abs(a) + (hi_binade(q) - ((1023 + 53) << 20))) && !pow2_significand(q);
}

__device__ __forceinline__ double rcp_estimate(const double a)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return y;
}

__device__ __forceinline__ double div_try(const double h, const double a, bool &ok)
{
  const double y0 = rcp_estimate(a), q0 = h * y0;
  const double e = __fma_rn(-a, y0, 1.0);
  const double y1 = __fma_rn(y0, e, y0), q1 = __fma_rn(q0, e, q0);
  const double q = __fma_rn(__fma_rn(-a, q1, h), y1, q1);
  ok = quotient_ok(__fma_rn(-a, q, h), a, q);
  return q;
}

__device__ __forceinline__ double rcp_try(const double a, bool &ok)
{
  const double y0 = rcp_estimate(a);
  const double y1 = __fma_rn(y0, __fma_rn(-a, y0, 1.0), y0);
  const double t = __fma_rn(__fma_rn(-a, y1, 1.0), y1, y1);
  ok = quotient_ok(__fma_rn(-a, t, 1.0), a, t);
  return t;
}

// sqrt(x): sqrt(x) and 1 / (2 sqrt(x)) to 2^-39 by one step, then the residual;
// s is sqrt(x) rounded to nearest if |x - s^2| < s ulp(s)
__device__ __forceinline__ double sqrt_try(const double x, bool &ok)
{
  const double y0 = rsqrt_estimate(x);
  const double g0 = x * y0, h0 = 0.5 * y0;
  const double r0 = __fma_rn(-g0, h0, 0.5);
  const double g1 = __fma_rn(g0, r0, g0), h1 = __fma_rn(h0, r0, h0);
  const double s = __fma_rn(__fma_rn(-g1, g1, x), h1, g1);
  const double rho = __fma_rn(-s, s, x);
  ok = (hi_abs(rho) < hi_abs(s) + (hi_binade(s) - ((1023 + 52) << 20))) && !pow2_significand(s);
  return s;
}

// 1 / sqrt(f), f = 1 +- t^2, by g = 1 - f (exact) for |g| < 2^-30: 1 + g (1/2 +
// 3/8 g) rounded once.  There 1 + g/2 is a representable number, a midpoint or a
// quarter of the spacing, and the true value lies above it by 3/8 g^2 + ...: the
// computed sum lies above it too (1/2 is taken one ulp larger, for the g whose
// 3/8 g is lost) and by less than a quarter of the spacing, so it rounds as the
// true value does; for g < 0 1 + g/2 is representable and both round to it.
__device__ __forceinline__ double rsqrt_near1(const double g, bool &ok)
{
  ok = hi_abs(g) < ((1023 - 30) << 20);
  return __fma_rn(g, __fma_rn(0.375, g, 0x1.0000000000001p-1), 1.0);
}

// rsqrt_rn: the fast path, and rsqrt_rn_full for what it does not settle
__device__ __forceinline__ bool rsqrt_range(const double a) // 2^-960 <= a < 2^960
{
  return (unsigned)(__double2hiint(a) - (63 << 20)) < (1920u << 20);
}

__device__ __forceinline__ double rsqrt_rn(const double a)
{
  bool ok;
  const double c = rsqrt_try(a, ok);
  return (ok && rsqrt_range(a)) ? c : rsqrt_rn_full(a);
}

// ---------------------------------------------------------------------------
// 32-lane butterfly sum (share/device_code_common_Kepler.hpp:26-74): lane i
// adds lane i^16, i^8, i^4, i^2, i^1; the result is lane 0's, broadcast.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double sum32(double v)
{
  v = v + __shfl_xor_sync(0xffffffffu, v, 16);
  v = v + __shfl_xor_sync(0xffffffffu, v, 8);
  v = v + __shfl_xor_sync(0xffffffffu, v, 4);
  v = v + __shfl_xor_sync(0xffffffffu, v, 2);
  v = v + __shfl_xor_sync(0xffffffffu, v, 1);
  return __shfl_sync(0xffffffffu, v, 0);
}

// ---------------------------------------------------------------------------
// 2x2 rotations (share/device_code_common_rotate.hpp:16-64, USE_RSQRT form):
// the three cases of each kind are selects of values that every lane
// computes, so the lanes that evaluate different rotations never diverge.
// "big" rotations (c != 1) are counted.
// ---------------------------------------------------------------------------
// one inner rotation, as the lanes that compute it hand it to those that apply it
struct Rot {
  double c, t, t_;
  int mode; // 0 nothing, 1 rotate, 2 swap columns
  int scale, swap;
};

// rotT for the lanes with trig, rotH for the others, in one chain, by the
// IEEE operations.  The two formulas take the same operations up to signs --
// Dq - Dp is Dq + (-Dp) exactly, the quotient negated, +1 or -1 under the
// square root, t t + 1 or -t t + 1 under the reciprocal square root -- and
// their special cases are selects, so each lane gets exactly the operations
// of its own formula while a warp whose lanes need both kinds runs one chain
// of divides and square roots instead of two.
__device__ __forceinline__ int rotTH(const bool trig, const double Apq, const double Dp, const double Dq, double &c,
                                     double &t)
{
  const double h = Dq + (trig ? -Dp : Dp);
  const double qt = __ddiv_rn(h, Apq * 2.0);
  const double ct2 = trig ? qt : -qt;
  const double CT2 = fabs(ct2);
  const bool large = CT2 >= kSqrt2Heps;
  const bool small = trig && (CT2 < kSqrtHeps);      // rotT's first case
  const bool mid = !trig && !large && (CT2 > 1.0);  // rotH's middle case
  const double cot_mid = CT2 + __dsqrt_rn(__fma_rn(CT2, CT2, trig ? 1.0 : -1.0));
  const double cot = small ? (CT2 + 1.0) : (large ? (CT2 * 2.0) : cot_mid);
  const double tt = copysign(__drcp_rn(cot), ct2);
  const double cr = rsqrt_rn(__fma_rn(trig ? tt : -tt, tt, 1.0));
  c = large ? 1.0 : ((trig || mid) ? cr : kCoshIFix);
  t = (trig || large || mid) ? tt : kTanh1Fix;
  return trig ? (small ? 1 : (large ? 0 : (cr < 1.0))) : (large ? 0 : (mid ? (cr > 1.0) : 1));
}

// the relative test and the rotation by the IEEE operations: the lanes whose
// fast path could not prove a value (c | t | ts | b)
struct RotRaw {
  double c, t;
  int ts, b;
};
static __device__ __noinline__ RotRaw rot_ieee(const bool trig, const double Apq, const double Dp, const double Dq)
{
  RotRaw r;
  r.ts = !(fabs(Apq) < ((__dsqrt_rn(Dp) * __dsqrt_rn(Dq)) * kMyTol));
  r.b = rotTH(trig, Apq, Dp, Dq, r.c, r.t);
  return r;
}

// The same values by the branch-free operations above, in one block of
// independent chains.  MIXED: some lanes of the warp are hyperbolic.
// The relative test |Apq| < RN(RN(sqrt Dp) RN(sqrt Dq)) tol is decided by Apq^2
// against Dp Dq tol^2 (tol^2 = 2^-101 to 2^-52), without the two square roots:
// the high words order as the rounded sides do when they differ by 2 or more
// (2^-20 relatively, the roundings 2^-49).
// Measured (inner_rot, one warp; two warps per sub-partition): 451 and 538
// cycles, against 715 and 775 with the IEEE operations one after the other.
// bad: a value that this lane's rotation uses is not proved, or the test is
// too close to call, or Dp Dq is outside 2^+-800 (within it no intermediate
// result above leaves the normal range unnoticed).  There (columns of norms below
// about 2^-200 or above 2^200) every rotation takes both ways: 2560^2 with entries
// of 2^+-300 ALG 9 177 ms, ALG 3 367, against 149 and 245 within the range and 194
// and 359 by the IEEE operations alone.  Remembering from step to step that a
// lane is out of range (168 and 334) costs calls within it 1 to 3 %.
template <bool MIXED>
__device__ __forceinline__ RotRaw rot_try(const bool trig, const double Apq, const double Dp, const double Dq,
                                          bool &bad)
{
  RotRaw r;
  const int hP = __double2hiint(Dp * Dq), dh = __double2hiint(Apq * Apq) - (hP - (101 << 20));
  const bool sure = ((unsigned)(hP - (223 << 20)) < (1600u << 20)) && ((unsigned)(dh + 1) > 2u);
  r.ts = dh > 0;

  const double h = Dq + ((!MIXED || trig) ? -Dp : Dp);
  bool ok_q, ok_s, ok_t, ok_c;
  const double qt = div_try(h, Apq * 2.0, ok_q);
  const double ct2 = (!MIXED || trig) ? qt : -qt;
  const double CT2 = fabs(ct2);
  const unsigned long long cbits = (unsigned long long)__double_as_longlong(CT2);
  const bool large = cbits >= (unsigned long long)__double_as_longlong(kSqrt2Heps);
  const bool small = (!MIXED || trig) && (cbits < (unsigned long long)__double_as_longlong(kSqrtHeps));
  const bool fixed = MIXED && !trig && (cbits <= 0x3FF0000000000000ull); // rotH's last case: constants
  const double alt = small ? 1.0 : CT2; // cot = CT2 + 1, 2 CT2 or CT2 + sqrt(CT2^2 +- 1)
  const double sq = sqrt_try(__fma_rn(CT2, CT2, (!MIXED || trig) ? 1.0 : -1.0), ok_s);
  const double t = rcp_try(CT2 + ((small || large) ? alt : sq), ok_t);
  const double f = __fma_rn((!MIXED || trig) ? t : -t, t, 1.0), g = 1.0 - f;
  const double cr = rsqrt_try(f, ok_c);
  bool near1;
  const double cn = rsqrt_near1(g, near1), c1 = near1 ? cn : cr;
  r.c = large ? 1.0 : (fixed ? kCoshIFix : c1);
  r.t = fixed ? kTanh1Fix : copysign(t, ct2);
  r.b = (unsigned long long)__double_as_longlong(r.c) != 0x3FF0000000000000ull; // c != 1
  bad = !sure || (r.ts && (!ok_q || (!fixed && (!ok_t || !(large || ((near1 || ok_c) && (small || ok_s)))))));
  return r;
}

template <bool SORT>
__device__ __forceinline__ Rot inner_rot(const double Dp, const double Dq, const double Apq, const unsigned p,
                                         const unsigned q, const int definite, const unsigned npos, unsigned &ts_out,
                                         unsigned &tb_out)
{
  // branch-free: the parts of a warp handle different pairs, so every choice
  // below is a select of values computed by both (no divergent paths); the
  // rotation is computed whether or not it is applied
  const int def = definite ? definite : ((p < npos) && (q < npos)) ? +1 : ((p >= npos) && (q >= npos)) ? -1 : 0;
  bool bad;
  RotRaw w = (definite || __all_sync(0xffffffffu, def != 0)) ? rot_try<false>(true, Apq, Dp, Dq, bad)
                                                             : rot_try<true>(def != 0, Apq, Dp, Dq, bad);
  if (bad)
    w = rot_ieee(def != 0, Apq, Dp, Dq);
  Rot r;
  const int ts = w.ts;
  const double t_ = def ? -w.t : w.t;
  r.c = ts ? w.c : 1.0;
  r.t = ts ? w.t : 0.0;
  r.t_ = ts ? t_ : 0.0;
  const int tb = ts ? w.b : 0;
  r.scale = tb;
  if (!SORT) {
    r.mode = ts;
    r.swap = 0;
  }
  else {
    const double Dp2 = __fma_rn(w.t, Apq, Dp), Dq2 = __fma_rn(t_, Apq, Dq); // used when ts and def
    const int swp = !((!def) || ((def > 0) && (Dp2 >= Dq2)) || ((def < 0) && (Dp2 <= Dq2)));
    const int order = ((def > 0) && (Dp < Dq)) || ((def < 0) && (Dq < Dp));
    r.mode = ts ? 1 : (order ? 2 : 0);
    r.swap = ts ? swp : 0;
  }
  ts_out = (unsigned)ts;
  tb_out = (unsigned)tb;
  return r;
}

// a named barrier for the nthreads threads of a warp group (id 0 with all the
// CTA's threads is __syncthreads)
__device__ __forceinline__ void bar_sync(const unsigned id, const unsigned nthreads)
{
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// programmatic dependent launch: let the next launch of the stream be placed
// (it waits in pdl_wait until this grid is complete and its writes visible);
// both do nothing in a launch without the attribute
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A CTA's shared memory may be accessed from its cluster once the CTA has
// started: every thread of every CTA arrives when it runs, and waits before the
// cluster's first remote store.  No data is handed over (relaxed).  Between the
// two lies the Gram phase, so nobody is waited for in practice.
__device__ __forceinline__ void cluster_started() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_started() { asm volatile("barrier.cluster.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------
// mbarrier + bulk-copy (TMA engine) helpers, with bounded waits
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, const uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_inval(uint64_t *bar)
{
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, const uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, const uint32_t parity)
{
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\t"
               "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return done != 0u;
}

// Wait for the phase with the given parity, at most ~limit_cycles.  Returns
// false on timeout (the caller records an error and stops waiting).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, const uint32_t parity,
                                                  const long long limit_cycles)
{
  if (mbar_try_wait(bar, parity))
    return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > limit_cycles)
      return false;
  }
  return true;
}

// 1-D bulk copy global -> shared, completing bytes on the mbarrier.
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, const uint32_t bytes, uint64_t *bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// 16-byte asynchronous copy global -> shared (both 16-byte aligned), L2 only
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// one arrival on the mbarrier once all prior cp.async of this thread completed
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar)
{
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// TMA tensor copy of a 3-D box at (c0, c1, c2) of the tensor map (kernel
// parameter space) into shared memory, completing bytes on the mbarrier.
// c0 * element size must be a multiple of 16 bytes (c0 = 0 here).
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *tm, const int c0, const int c1,
                                            const int c2, uint64_t *bar)
{
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
               "[%5];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
               : "memory");
}

// TMA tensor store of a 3-D box of shared memory to (c0, c1, c2) of the
// tensor map, in this thread's current bulk async-group; elements of the box
// outside the tensor are not written.  c0 = 0 here; no coordinate is negative.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *tm, const void *src, const int c0, const int c1,
                                             const int c2)
{
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tm)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// 1-D bulk copy shared -> global in this thread's current bulk async-group;
// dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, const uint32_t bytes)
{
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

// close this thread's bulk async-group
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

// this thread's bulk groups have finished reading shared memory
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// all but this thread's most recent bulk group have finished reading shared memory
__device__ __forceinline__ void bulk_wait_read_but1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }

// this thread's bulk groups are complete (their global writes performed),
// and ordered before this thread's later generic-proxy operations
__device__ __forceinline__ void bulk_wait_all()
{
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

// this thread's shared-memory writes become visible to the async proxy (a TMA
// store issued after a barrier)
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

} // namespace gjx
