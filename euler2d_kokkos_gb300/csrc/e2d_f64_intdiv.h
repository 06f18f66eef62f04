// e2d_f64_intdiv.h -- correctly rounded FP64 division and square root in
// integer arithmetic.
//
// GB300 runs one FP64 warp instruction per SM and 16 clocks (three-register
// FMAs; 19 for any other form, see Fp in e2d_f64_exact.cuh), and an IEEE
// division or square root is a sequence of about nine of them: 580 clocks per
// warp and scheduler, measured.  The integer pipes are idle meanwhile.  The
// quotient below takes 85 clocks (103 for the square root) and no FP64
// instruction at all, and it overlaps with FP64 arithmetic: four FMAs and one
// quotient take as long as the four FMAs alone (GB300, 8 blocks of 256
// threads per SM).
//
// Method: schoolbook long division with two large digits.  A 32-bit
// reciprocal estimate of the divisor that never exceeds the true value (the
// FP32 reciprocal plus one Newton-Raphson step on integers) gives a 32-bit
// digit, the exact remainder gives a 27-bit one, and one comparison makes the
// 54- or 55-bit quotient the exact floor.  A quotient of two 53-bit
// significands cannot lie halfway between two neighbouring doubles, so adding
// half a unit to the floor and truncating rounds to nearest.  The square root
// goes the same way with the reciprocal square root, digit by digit
// (remainder x - s^2).  Results equal the IEEE operation's bit for bit.
//
// Compiles for the host too (tests), where the seeds come from FP32 division.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define E2D_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define E2D_HD inline
#endif

namespace e2d {
namespace f64i {

E2D_HD uint32_t mul_hi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// high word of (hi:lo) << s, 0 < s < 32
E2D_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (hi << s) | (lo >> (32 - s));
#endif
}
// The words of a double.  On the device by a PTX move: the compiler turns
// sign and magnitude tests of a bit pattern it knows to be a double's back
// into FP64 instructions (measured: 34 of the slopes' 58 per cell).
E2D_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  uint64_t b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
E2D_HD double make(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  double d;
  asm("mov.b64 %0, {%1, %2};" : "=d"(d) : "r"(lo), "r"(hi));
  return d;
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double d;
  std::memcpy(&d, &b, 8);
  return d;
#endif
}
E2D_HD uint32_t high(double x) {
#ifdef __CUDA_ARCH__
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
  return hi;
#else
  return (uint32_t)(bits(x) >> 32);
#endif
}
E2D_HD uint32_t low(double x) {
#ifdef __CUDA_ARCH__
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
  return lo;
#else
  return (uint32_t)bits(x);
#endif
}
// x > 0.0 (a NaN of either sign gives false)
E2D_HD bool positive(double x) { return bits(x) - 1u < 0x7ff0000000000000ull; }
// FP32 seeds: bit patterns of 1 / f, f in [1, 2), and 1 / sqrt(f), f in [1, 4).
// They may exceed the true value by 4 and 3 units of 2^-24 at most: divisor()
// lowers the reciprocal by 6, of which dropping b's low bits takes up to 2
// (2^-23 / b^2), root() its seed by 4, of which they take up to 1; a seed that
// stays above 1 / b makes wrong quotients that `ok` does not show.  The
// instructions are specified within 2^-23 and 2^-22.9 (2 and 2.1 units).  The
// tests sweep every seed the device can give, and the host's moved by 2 units
// (E2D_SEED_SHIFT).
#ifndef E2D_SEED_SHIFT
#define E2D_SEED_SHIFT 0
#endif
E2D_HD uint32_t seed_rcp(uint32_t f) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return __float_as_uint(y);
#else
  float x;
  std::memcpy(&x, &f, 4);
  x = 1.0f / x;
  std::memcpy(&f, &x, 4);
  return f + (uint32_t)(E2D_SEED_SHIFT);
#endif
}
E2D_HD uint32_t seed_rsqrt(uint32_t f) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return __float_as_uint(y);
#else
  float x;
  std::memcpy(&x, &f, 4);
#ifdef __CUDACC__
  x = (float)(1.0 / sqrt((double)x));
#else
  x = (float)(1.0 / std::sqrt((double)x));
#endif
  std::memcpy(&f, &x, 4);
  return f + (uint32_t)(E2D_SEED_SHIFT);
#endif
}

// A divisor made ready for one or several quotients: its words and the
// reciprocal estimate y <= 2^32 / b, b in [1, 2) its significand, short of it
// by less than 2^-28.6 relative (checked over every leading 24 bits).
struct Divisor {
  uint32_t hi, lo, y;
};

E2D_HD Divisor divisor(double d) {
  Divisor v;
  v.hi = high(d);
  v.lo = low(d);
  const uint32_t bt = shl_hi(v.lo, (v.hi & 0xfffffu) | 0x100000u, 11);  // b 2^31, truncated
  // FP32 reciprocal of b's leading 24 bits, y in (1/2, 1], as a 32-bit
  // fraction lowered by 6 units of its last place so that it stays below 1/b
  const uint32_t y0 = (seed_rcp((bt >> 8) + 0x3f000000u) << 8) + (0x80000000u - 1536u);
  // Newton: y1 = y0 + y0 (1 - b y0), lowered by the four truncations' units
  const uint32_t e = 0u - 2u * mul_hi(bt, y0);
  v.y = y0 + mul_hi(y0, e) - 4u;
  return v;
}

// a / d rounded to nearest for d in [2^-500, 2^501), a zero or normal, and a
// normal result; otherwise `ok` is false and the value is meaningless.
E2D_HD double quotient(double a, const Divisor &d, bool &ok) {
  const uint32_t ah = high(a), al = low(a);
  const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, b1 = (d.hi & 0xfffffu) | 0x100000u;
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (d.hi >> 20) & 0x7ffu;
  const uint64_t A = ((uint64_t)a1 << 32) | al;  // significands, 53 bits
  const uint64_t B = ((uint64_t)b1 << 32) | d.lo;
  // digit 1: 2^31 a/b less at most 7; remainder < 8 B, exact modulo 2^64
  const uint32_t q1 = mul_hi(shl_hi(al, a1, 11), d.y);
  const uint64_t r1 = (A << 31) - ((uint64_t)q1 * d.lo + ((uint64_t)(q1 * b1) << 32));
  // digit 2: 23 more bits of it, less at most 1
  const uint32_t q2 = mul_hi((uint32_t)(r1 >> 25), d.y) >> 4;
  const uint64_t r2 = (r1 << 23) - ((uint64_t)q2 * d.lo + ((uint64_t)(q2 * b1) << 32));
  const uint64_t q = (uint64_t)q1 * (1u << 23) + (q2 + (r2 >= B ? 1u : 0u));  // floor(2^54 a/b)
  // round to 53 bits; c: a/b >= 1, one bit more to drop
  const uint32_t c = (uint32_t)(q >> 54);
  const uint64_t m = (q + (1u << c)) >> (1u + c);
  const uint32_t er = ea - eb + 1021u + c;  // m's leading bit carries into it
  const uint32_t sign = (ah ^ d.hi) & 0x80000000u;
  const bool zero = ((ah & 0x7fffffffu) | al) == 0u;
  ok = eb - 523u < 1001u && ((ea - 1u < 2046u && er < 2045u) || zero);
  const uint32_t rh = (uint32_t)(m >> 32) + (er << 20);
  return make(zero ? sign : (sign | rh), zero ? 0u : (uint32_t)m);
}

// sqrt(x) rounded to nearest for x in [2^-500, 2^501); otherwise `ok` is
// false and the value is meaningless.
E2D_HD double root(double x, bool &ok) {
  const uint32_t xh = high(x), xl = low(x);
  const uint32_t ex = xh >> 20;       // the sign is clear when ok
  const uint32_t odd = ~ex & 1u;      // exponent ex - 1023 odd: m in [2, 4)
  const uint32_t m1 = (xh & 0xfffffu) | 0x100000u;
  const uint64_t M = (((uint64_t)m1 << 32) | xl) << odd;  // m 2^52, m in [1, 4)
  const uint32_t mt = (uint32_t)(M >> 22);                // m 2^30, truncated
  const uint32_t f = (shl_hi(xl, m1, 3) & 0x7fffffu) | (0x3f800000u + (odd << 23));
  const uint32_t y0 = (seed_rsqrt(f) << 8) + (0x80000000u - 1024u);  // 2^32 / sqrt(m), from below
  const uint32_t e = 0x40000000u - mul_hi(mt, mul_hi(y0, y0));       // 2^30 (1 - m y0^2) >= 0
  const uint32_t y = y0 + mul_hi(y0, e << 1) - 6u;                   // Newton: y0 + y0 (1 - m y0^2) / 2
  // digit 1: 2^30 sqrt(m) less at most 8; digit 2: 23 more bits, less at most 1
  const uint32_t s1 = mul_hi(mt, y);
  const uint64_t r1 = (M << 8) - (uint64_t)s1 * s1;
  const uint32_t s2 = mul_hi((uint32_t)(r1 >> 4), y) >> 4;
  // remainder of (s1 2^23 + s2)^2, exact modulo 2^64
  const uint64_t w = ((uint64_t)s1 << 24) + s2;
  const uint64_t r2 = (r1 << 46) - ((uint64_t)s2 * (uint32_t)w + ((uint64_t)(s2 * (uint32_t)(w >> 32)) << 32));
  const uint64_t s = ((uint64_t)s1 << 23) + s2;
  const uint64_t m2 = (s + (r2 > 2u * s ? 2u : 1u)) >> 1;  // floor(2^53 sqrt(m)), rounded to 53 bits
  const uint32_t er = ((ex + 1023u - odd) >> 1) - 1u;      // m2's leading bit carries into it
  ok = ex - 523u < 1001u;
  return make((uint32_t)(m2 >> 32) + (er << 20), (uint32_t)m2);
}

// a * b rounded to nearest even for normal a, b and a normal result;
// otherwise `ok` is false and the value is meaningless.
E2D_HD double product(double a, double b, bool &ok) {
  const uint32_t ah = high(a), al = low(a), bh = high(b), bl = low(b);
  const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, b1 = (bh & 0xfffffu) | 0x100000u;
  // the 106-bit product of the significands: t3 (42 bits), t2, t0 (low words)
  const uint64_t t0 = (uint64_t)al * bl;
  const uint64_t t1 = (uint64_t)a1 * bl + (t0 >> 32);
  const uint64_t t2 = (uint64_t)al * b1 + t1;
  const uint64_t t3 = (uint64_t)a1 * b1 + (t2 >> 32);
  const uint32_t c = (uint32_t)(t3 >> 41);  // 1: the product is in [2, 4)
  // 53 + c bits and a 32-bit fraction whose last bit is sticky
  const uint32_t mh = shl_hi((uint32_t)t3, (uint32_t)(t3 >> 32), 12), ml = shl_hi((uint32_t)t2, (uint32_t)t3, 12);
  const uint32_t s = ((uint32_t)t2 << 12) | ((uint32_t)t0 != 0u ? 1u : 0u);
  const uint64_t m = (((uint64_t)mh << 32) | ml) >> c;
  const uint32_t f = (uint32_t)((((uint64_t)ml << 32) | s) >> c) | (s & c);
  const uint64_t r = m + ((f >> 31) & (uint32_t)((f << 1) != 0u || (m & 1u)));
  const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  const uint32_t e = ea + eb + (c << 20) - (1024u << 20);  // m's leading bit carries into it
  const bool zero = ((ah & 0x7fffffffu) | al) == 0u || ((bh & 0x7fffffffu) | bl) == 0u;
  ok = zero ? (ea != 0x7ff00000u && eb != 0x7ff00000u)
            : (ea - 0x00100000u < 0x7fe00000u && eb - 0x00100000u < 0x7fe00000u && e < 0x7fd00000u);
  return make((zero ? 0u : (uint32_t)(r >> 32) + e) | ((ah ^ bh) & 0x80000000u), zero ? 0u : (uint32_t)r);
}

}  // namespace f64i
}  // namespace e2d
