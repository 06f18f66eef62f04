// e2d_f64_exact.cuh -- exact FP64 operations carried out on the integer
// pipe.
//
// GB300 issues FP64 arithmetic at 1.7 to 2 operations per SM per clock, about
// 1/64 of its FP32 rate.  Comparisons, min/max against known signs, sign
// tests and multiplications by 0.5 or 2 do not need the FP64 unit: on the
// bit patterns of IEEE-754 doubles they are integer operations that give the
// same bits as the FP64 instructions.  Each helper states the inputs for which
// that holds; outside them (NaN, subnormal results) it falls back to the FP64
// instruction itself, so results stay bit-identical to the plain expression.
#pragma once

#include <cuda_runtime.h>

#include "e2d_f64_intdiv.h"

namespace e2d {
namespace f64x {

constexpr unsigned long long kMag = 0x7fffffffffffffffull;
constexpr unsigned long long kSign = 0x8000000000000000ull;

__device__ __forceinline__ unsigned long long ubits(double x) { return f64i::bits(x); }
__device__ __forceinline__ long long sbits(double x) { return (long long)f64i::bits(x); }
__device__ __forceinline__ double from_bits(unsigned long long b) {
  return f64i::make((uint32_t)(b >> 32), (uint32_t)b);
}

// a / b and sqrt(x) as the IEEE operations give them, on the integer pipes
// (e2d_f64_intdiv.h); operands outside their range run the operation itself.
static __device__ __noinline__ double div_slow(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_slow(double x) { return sqrt(x); }
using f64i::Divisor;
using f64i::divisor;
__device__ __forceinline__ double quot(double a, const Divisor &d) {
  bool ok;
  double q = f64i::quotient(a, d, ok);
  if (!ok) q = div_slow(a, f64i::make(d.hi, d.lo));
  return q;
}
__device__ __forceinline__ double quot(double a, double b) { return quot(a, divisor(b)); }
__device__ __forceinline__ double root(double x) {
  bool ok;
  double s = f64i::root(x, ok);
  if (!ok) s = sqrt_slow(x);
  return s;
}

// FP64 multiply kept out of line so that it runs only on the lanes that need
// it (a branch, not a predicated instruction issued by the whole warp).
static __device__ __noinline__ double mul_slow(double a, double b) { return a * b; }

// fmax(x, c) for c > 0: non-negative doubles order like their bit patterns as
// signed integers and every negative x (including -0) is below c.
// (NaN x is returned instead of c; NaN states are flagged elsewhere.)
__device__ __forceinline__ double max_pos(double x, double c) { return sbits(x) > sbits(c) ? x : c; }

// fmax / fmin of two non-negative doubles.
__device__ __forceinline__ double max_nn(double a, double b) { return sbits(a) > sbits(b) ? a : b; }
__device__ __forceinline__ double min_nn(double a, double b) { return sbits(a) < sbits(b) ? a : b; }

// fmin / fmax of two doubles of any sign: the key flips the magnitude bits of
// negatives so that keys order like the values; -0 orders below +0 (either
// is a valid fmin(+0, -0)).
__device__ __forceinline__ long long okey(double x) {
  const long long b = sbits(x);
  return b ^ ((b >> 63) & (long long)kMag);
}
__device__ __forceinline__ double min_any(double a, double b) { return okey(a) <= okey(b) ? a : b; }
__device__ __forceinline__ double max_any(double a, double b) { return okey(a) >= okey(b) ? a : b; }

// Sign tests for non-NaN x.
__device__ __forceinline__ bool gt0(double x) { return sbits(x) > 0; }   // x > 0.0
__device__ __forceinline__ bool le0(double x) { return sbits(x) <= 0; }  // x <= 0.0
__device__ __forceinline__ bool lt0(double x) { return (ubits(x) > kSign) & (sbits(x) < 0); }  // x < 0.0
__device__ __forceinline__ bool is_nan(double x) { return (ubits(x) & kMag) > 0x7ff0000000000000ull; }
// x > c for x >= 0 and c > 0 (a NaN x gives false)
__device__ __forceinline__ bool gt_pos(double x, double c) { return sbits(x) > sbits(c) && !is_nan(x); }

// 0.5 * x: decrement the exponent of normal numbers with a biased exponent in
// [2, 2046]; zeros are unchanged; subnormal results need rounding and use the
// FP64 multiply; Inf/NaN are unchanged.
__device__ __forceinline__ double half(double x) {
  const int hi = (int)f64i::high(x);
  const int lo = (int)f64i::low(x);
  const int e = (hi >> 20) & 0x7ff;
  if (e >= 2 && e < 0x7ff) return f64i::make((uint32_t)hi - 0x00100000u, (uint32_t)lo);
  if (((hi & 0x7fffffff) | lo) == 0 || e == 0x7ff) return x;
  return mul_slow(0.5, x);
}

// 2.0 * x: increment the exponent of normal numbers below 2^1023 ...; zeros
// unchanged; subnormals and overflow use the FP64 multiply.
__device__ __forceinline__ double twice(double x) {
  const int hi = (int)f64i::high(x);
  const int lo = (int)f64i::low(x);
  const int e = (hi >> 20) & 0x7ff;
  if (e >= 1 && e < 0x7fe) return f64i::make((uint32_t)hi + 0x00100000u, (uint32_t)lo);
  if (((hi & 0x7fffffff) | lo) == 0 || e == 0x7ff) return x;
  return mul_slow(2.0, x);
}

// Additions and products as fused multiply-adds of three registers.  The FP64
// pipe takes 16 clocks per SM for a warp's DFMA whose operands are all
// registers and 19 for a DADD, a DMUL or any form with a constant or uniform
// operand (measured: 625 against 527 G operations/s), so x + y is issued as
// x * 1 + y, x - y as y * (-1) + x and x * y as x * y + (-0): the same
// roundings and the same signs of zero.  1 and -0 have to sit in registers the compiler knows nothing of;
// each lane loads them from its own address.
static __device__ double2 g_unit[32] = {
#define E2D_U4 {1.0, -0.0}, {1.0, -0.0}, {1.0, -0.0}, {1.0, -0.0}
    E2D_U4, E2D_U4, E2D_U4, E2D_U4, E2D_U4, E2D_U4, E2D_U4, E2D_U4
#undef E2D_U4
};
//
// XMUL: xmul() forms the product on the integer pipes (35 instructions, about
// 60 clocks, overlapping the FP64 pipe's 64).  With about a fifth of a step's
// products there the two pipes run side by side.  HLLC: face increments,
// transport terms, contact sums, energies, flux scaling, 1.556 instead of 1.69
// ms a 2048^2 step; with more of them the step slows down again (1.57 to 1.63
// ms).  HLL: energies, transverse momentum and energy fluxes, jump
// terms and the final scaling, 1.866 -> 1.761 ms with tiles, 1.574 -> 1.548
// for the scaling (march).  The fast forms, which have the fewest FP64 instructions: all
// products that are not part of an FMA, 1.308 -> 1.236 ms.  Where each SM holds
// one small tile the step waits on latency, not on the FP64 pipe, and the
// plain product is the faster one (64x48: 16.0 against 17.1 us a step).
template <bool XMUL>
struct FpT {
  double one, mzero, mone;
  __device__ __forceinline__ FpT() {
    const double2 *p = g_unit + (threadIdx.x & 31);
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(one), "=d"(mzero) : "l"(p));
    mone = neg(one);
  }
  // sign changes on the integer pipe: a negated FP64 operand that several
  // instructions read is otherwise formed by an FP64 instruction of its own
  static __device__ __forceinline__ double neg(double x) {
    return f64i::make(f64i::high(x) ^ 0x80000000u, f64i::low(x));
  }
  static __device__ __forceinline__ double abs(double x) {
    return f64i::make(f64i::high(x) & 0x7fffffffu, f64i::low(x));
  }
  // -x where x is a difference a - b: b - a (+0, not -0, where they are equal)
  static __device__ __forceinline__ double reversed(double x) {
    const unsigned int hi = f64i::high(x), lo = f64i::low(x);
    return f64i::make(((hi << 1) | lo) != 0u ? hi ^ 0x80000000u : 0u, lo);
  }
  __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
  __device__ __forceinline__ double sub(double a, double b) const { return fma(b, mone, a); }
  __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, mzero); }
  __device__ __forceinline__ double xmul(double a, double b) const {
    if (!XMUL) return mul(a, b);
    bool ok;
    double p = f64i::product(a, b, ok);
    if (!ok) p = mul_slow(a, b);
    return p;
  }
  // 0.5 * (a * b) given hb = 0.5 * b: one product, unless halving would round
  // (a result below the smallest normal double)
  __device__ __forceinline__ double half_product(double a, double b, double hb) const {
    if (XMUL) return half(xmul(a, b));
    double p = mul(a, hb);
    if ((f64i::high(p) & 0x7ff00000u) == 0u && ((f64i::high(a) & 0x7fffffffu) | f64i::low(a)) != 0u)
      p = mul_slow(0.5, mul_slow(a, b));
    return p;
  }
};
using Fp = FpT<true>;

// src/HydroBaseFunctor.h:421-455, one direction, for slope_type st in {1, 2}:
//   dlft = st*(q-qm); drgt = st*(qp-q); dcen = 0.5*(qp-qm)
//   dsgn = dcen >= 0 ? 1 : -1; slop = fmin(|dlft|, |drgt|)
//   dlim = (dlft*drgt <= 0) ? 0 : slop;  dq = dsgn * fmin(dlim, |dcen|)
// from the three differences, as written.
static __device__ __noinline__ double limit_slow(bool st2, double d1, double d2, double dc) {
  const double st = st2 ? 2.0 : 1.0;
  const double dl = mul_slow(st, d1), dr = mul_slow(st, d2), dcen = mul_slow(0.5, dc);
  const double slop = fmin(fabs(dl), fabs(dr));
  const double dlim = (dl * dr <= 0.0) ? 0.0 : slop;
  const double r = fmin(dlim, fabs(dcen));
  return dcen >= 0.0 ? r : -r;
}

// The same on the integer pipe but for the three differences.  The product
// test is "a zero or opposite signs" (the product underflows only below
// 2^-511); of one sign, the differences' sum dc has it too and is at least as
// large as either, so scaling by 2 and by 0.5 moves only the exponents.
// Differences outside [2^-511, 2^1023) that are not zero take the form above.
// h: dq / 2, which the face states need (exact: 0 or at least 2^-512).
template <class F>
__device__ __forceinline__ void slope_limited(const F &f, bool st2, double q, double qp, double qm, double &dq,
                                              double &h) {
  const double d1 = f.sub(q, qm);
  const double d2 = f.sub(qp, q);
  const double dc = f.sub(qp, qm);
  const unsigned int h1 = f64i::high(d1), h2 = f64i::high(d2), hc = f64i::high(dc), lc = f64i::low(dc);
  const unsigned long long a1 = ((unsigned long long)(h1 & 0x7fffffffu) << 32) | f64i::low(d1);
  const unsigned long long a2 = ((unsigned long long)(h2 & 0x7fffffffu) << 32) | f64i::low(d2);
  const unsigned long long m = a1 < a2 ? a1 : a2;
  const unsigned int mh = (unsigned int)(m >> 32), ac = hc & 0x7fffffffu;
  const bool mz = m == 0ull, cz = (ac | lc) == 0u;
  if ((mh < 0x20000000u && !mz) || (ac - 0x00200000u >= 0x7fc00000u && !cz)) {
    dq = limit_slow(st2, d1, d2, dc);
    h = 0.5 * dq;
    return;
  }
  // min(st m, |dc| / 2), halved once more below
  const unsigned long long lim = m + (st2 ? 1ull << 52 : 0ull);
  const unsigned long long cen = (((unsigned long long)ac << 32) | lc) - (1ull << 52);
  unsigned long long r = lim < cen ? lim : cen;
  const bool kill = mz || (int)(h1 ^ h2) < 0;
  const unsigned int sg = cz ? 0u : hc & 0x80000000u;  // dcen < 0
  const unsigned int rh = (unsigned int)(r >> 32), rl = kill ? 0u : (unsigned int)r;
  dq = f64i::make(sg | (kill ? 0u : rh), rl);
  h = f64i::make(sg | (kill ? 0u : rh - 0x00100000u), rl);
}

}  // namespace f64x
}  // namespace e2d
