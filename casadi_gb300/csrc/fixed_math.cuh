// Division, square root, sin/cos, exp, log and tanh of doubles in integer arithmetic.
//
// GB300 issues one FP64 warp instruction per sub-partition every 64 to 76 cycles, and about one
// integer instruction per cycle. Division costs 11 FP64 instructions, sincos 29, exp 21, log 35,
// tanh 17 (op_weights.json), i.e. 700 to 2400 cycles of the FP64 pipe each; the routines here
// take 55 to 200 integer instructions, run beside the pipe's additions and products, and shorten
// the dependent chain of one instance as well (an FP64 result takes 64 cycles, an integer one 4).
//
// * fx_div, fx_rcp, fx_sqrt return the correctly rounded result: a quotient (root) digit by
//   digit from a 31-bit reciprocal (Newton from a single-precision seed), the last bit settled
//   by the exact remainder. Neither a quotient nor a root of doubles lies halfway between two
//   doubles, so one more bit than the result and no sticky bit decides the rounding.
// * fx_sincos, fx_exp, fx_log, fx_tanh evaluate in 64-bit fixed point: argument reduction by a
//   96-bit constant, Chebyshev interpolants of the functions with the coefficients' and products'
//   width matched to their weight (errors below 2^-57), one rounding to double at the end. Largest
//   error against 113-bit references over 8 million arguments a range (CUDA's function beside it, over
//   2 million): sin and cos 0.505 ulp up to 3.2 (1.39), up to 100 (1.47) and up to 2^15, 0.544 next to
//   multiples of pi/2, exp 0.540 (0.864), log 0.533 (0.547), tanh 0.612 (1.42), just above 1/8, where
//   the quotient takes over from the series with its smallest result; 0.57 from 0.13 on.
//
// Arguments outside a routine's range (subnormals, infinities, NaN, zero numerators, quotients near
// the ends of the exponent range, huge arguments) make it return false: what it left in the result is
// not one. The caller settles zeros, infinities, NaN, overflow and underflow and takes CUDA's function
// for the rest (slow_* in device_ops.cuh), the whole warp for one such lane.
//
// Plain C++ apart from the seeds and the high products, so the routines can be compiled and
// checked on the host.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CGB_FX __host__ __device__ __forceinline__
#else
#include <math.h>
#define CGB_FX inline
#endif

namespace cgb {

typedef uint32_t fx_u32;
typedef uint64_t fx_u64;

CGB_FX fx_u64 fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<fx_u64>(__double_as_longlong(x));
#else
  fx_u64 b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
CGB_FX double fx_dbl(fx_u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(b));
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
CGB_FX fx_u32 fx_fbits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  fx_u32 b;
  memcpy(&b, &x, 4);
  return b;
#endif
}
CGB_FX float fx_flt(fx_u32 b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, 4);
  return x;
#endif
}
// Seeds: 1/x and 1/sqrt(x) to single precision (1 or 2 ulp)
CGB_FX float fx_rcp_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
CGB_FX float fx_rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / sqrtf(x);
#endif
}
CGB_FX fx_u32 fx_mulhi32(fx_u32 a, fx_u32 b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return static_cast<fx_u32>((static_cast<fx_u64>(a) * b) >> 32);
#endif
}
CGB_FX int fx_clz64(fx_u64 v) {
#ifdef __CUDA_ARCH__
  return __clzll(static_cast<long long>(v));
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
// High 64 bits of a*b without the low halves' product: at most 3 below floor(a*b / 2^64)
CGB_FX fx_u64 fx_mulhi(fx_u64 a, fx_u64 b) {
  const fx_u32 ah = static_cast<fx_u32>(a >> 32), al = static_cast<fx_u32>(a);
  const fx_u32 bh = static_cast<fx_u32>(b >> 32), bl = static_cast<fx_u32>(b);
  return static_cast<fx_u64>(ah) * bh + fx_mulhi32(ah, bl) + fx_mulhi32(al, bh);
}
CGB_FX fx_u32 fx_shf(fx_u32 lo, fx_u32 hi, int s) {  // high word of (hi:lo) << s, 0 <= s < 32
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

constexpr fx_u64 kFxSign = 0x8000000000000000ull;
constexpr fx_u64 kFxOne = 1ull << 52;
constexpr fx_u64 kFxMant = kFxOne - 1;

CGB_FX int fx_expo(fx_u64 b) { return static_cast<int>((b >> 52) & 0x7ffu); }

// The double of sign bit `sign` whose magnitude is v * 2^(expo - 1023 - 63): v normalised (top
// bit set), rounded to nearest.
CGB_FX double fx_pack(fx_u64 v, int expo, fx_u64 sign) {
  const fx_u64 m = (v >> 11) + ((v >> 10) & 1u);
  return fx_dbl((m + (static_cast<fx_u64>(static_cast<unsigned>(expo - 1)) << 52)) | sign);
}

// ---- reciprocals --------------------------------------------------------------------------------
// About 2^32 / y for a mantissa whose top 32 bits are yh (y = yh / 2^31 in [1, 2)): one Newton
// step from the single-precision seed, relative error within 2^-29.7; never above 2^32 - 1.
CGB_FX fx_u32 fx_rcp31(fx_u32 yh) {
  const fx_u32 f = fx_fbits(fx_rcp_seed(fx_flt(0x3f800000u | ((yh >> 8) & 0x7fffffu))));
  const fx_u32 c = f < 0x3f7fffffu ? f : 0x3f7fffffu;  // below 1
  const fx_u32 r0 = (c << 8) | 0x80000000u;
  const int e = static_cast<int>(0x80000000u - fx_mulhi32(r0, yh));
  return r0 + static_cast<fx_u32>((static_cast<int64_t>(r0) * e) >> 31);
}
// About 2^64 / d for d = dn / 2^63 in [1, 2): a second Newton step, from below (never above
// 2^64 - 1), relative error within 2^-58
CGB_FX fx_u64 fx_rcp62(fx_u64 dn) {
  const fx_u32 r = fx_rcp31(static_cast<fx_u32>(dn >> 32));
  const fx_u64 t = static_cast<fx_u64>(r) * static_cast<fx_u32>(dn >> 32) +
                   fx_mulhi32(r, static_cast<fx_u32>(dn));
  // t <= r*d, at most 1 below it (2^63: one); rounded up here so that the step stays below
  const int64_t e = static_cast<int64_t>(kFxSign - t) - 1;
  const int64_t c = (static_cast<int64_t>(e >> 4) * static_cast<int64_t>(r >> 1)) >> 26;
  return (static_cast<fx_u64>(r) << 32) + static_cast<fx_u64>(c) ;
}

// Rounded quotient bits of x / y from the mantissas mx, my (53 bits) and r = fx_rcp31(my >> 21):
// the 53-bit mantissa, leading bit set; *below is 1 when mx < my (the quotient is below 1).
CGB_FX fx_u64 fx_quot(fx_u64 mx, fx_u64 my, fx_u32 r, int* below) {
  const int c = mx < my ? 1 : 0;
  const fx_u64 x = mx << c;  // x / my in [1, 2)
  // 27 bits of the quotient, low by at most 1.2, high by at most 0.2
  const fx_u32 q1 = fx_mulhi32(static_cast<fx_u32>(x >> 22), r) >> 4;
  const int64_t rem1 = static_cast<int64_t>((x << 26) - static_cast<fx_u64>(q1) * my);
  // 27 more from the remainder
  const int q2 = static_cast<int>(
      (static_cast<int64_t>(static_cast<int>(rem1 >> 23)) * static_cast<int>(r >> 1)) >> 33);
  int64_t rem2 = static_cast<int64_t>((static_cast<fx_u64>(rem1) << 27) -
                                      static_cast<fx_u64>(static_cast<int64_t>(q2)) * my);
  fx_u64 q = (static_cast<fx_u64>(q1) << 27) + static_cast<fx_u64>(static_cast<int64_t>(q2));
  // floor(x / my * 2^53): the exact remainder is in [0, my)
  if (rem2 < 0) {
    q -= 1;
  } else if (rem2 >= static_cast<int64_t>(my)) {
    q += 1;
  }
  *below = c;
  return (q + 1) >> 1;
}

// Reciprocal data of a divisor, shared by several quotients.
struct FxDivisor {
  fx_u64 m;    // mantissa, 53 bits
  fx_u64 b;    // bits
  fx_u32 r;    // fx_rcp31
  int e;       // exponent field; 0 or 2047: not for these routines
};
CGB_FX FxDivisor fx_divisor(double y) {
  FxDivisor d;
  d.b = fx_bits(y);
  d.e = fx_expo(d.b);
  d.m = (d.b & kFxMant) | kFxOne;
  d.r = fx_rcp31(static_cast<fx_u32>(d.m >> 21));
  return d;
}
// x / y rounded to nearest; false when x, y or the quotient is not a normal number well inside the
// exponent range.
CGB_FX bool fx_div(double x, const FxDivisor& y, double* q) {
  const fx_u64 b = fx_bits(x);
  const int ex = fx_expo(b);
  int c;
  const fx_u64 m = fx_quot((b & kFxMant) | kFxOne, y.m, y.r, &c);
  const int e = ex - y.e + 1023 - c;
  *q = fx_dbl((m + (static_cast<fx_u64>(static_cast<unsigned>(e - 1)) << 52)) |
              ((b ^ y.b) & kFxSign));
  return static_cast<unsigned>(ex - 1) < 2046u && static_cast<unsigned>(y.e - 1) < 2046u &&
         static_cast<unsigned>(e - 1) < 2045u;
}

// sqrt(x) rounded to nearest, for normal positive x and zeros.
CGB_FX bool fx_sqrt(double x, double* s) {
  const fx_u64 b = fx_bits(x);
  if ((b << 1) == 0) {
    *s = x;
    return true;
  }
  const int ex = static_cast<int>(b >> 52);  // sign included: negative x fails the range check
  const int odd = (ex & 1) ^ 1;              // (ex - 1023) odd
  const fx_u64 a = ((b & kFxMant) | kFxOne) << odd;  // a / 2^52 in [1, 4)
  const fx_u32 ah = static_cast<fx_u32>(a >> 22);    // / 2^30
  const float af = fx_flt((odd ? 0x40000000u : 0x3f800000u) |
                          static_cast<fx_u32>((b >> 29) & 0x7fffffu));
  const fx_u32 f = fx_fbits(fx_rsqrt_seed(af));
  const fx_u32 cl = f < 0x3f7fffffu ? f : 0x3f7fffffu;
  const fx_u32 r0 = (cl << 8) | 0x80000000u;  // 2^32 / sqrt(a): in [1/2, 1)
  const int e = static_cast<int>(0x40000000u - fx_mulhi32(fx_mulhi32(r0, r0), ah));
  const fx_u32 r = r0 + static_cast<fx_u32>((static_cast<int64_t>(r0) * e) >> 31);
  // 27 bits of the root, then 27 more from the remainder a - s1^2
  const fx_u32 s1 = (fx_mulhi32(ah, r) + 8u) >> 4;
  const int64_t rem1 = static_cast<int64_t>(a - static_cast<fx_u64>(s1) * s1);
  const int q2 = static_cast<int>((rem1 * static_cast<int64_t>(r >> 1)) >> 31);
  int64_t rem2 = static_cast<int64_t>(
      (static_cast<fx_u64>(rem1) << 54) -
      static_cast<fx_u64>(static_cast<int64_t>(q2)) *
          ((static_cast<fx_u64>(s1) << 28) + static_cast<fx_u64>(static_cast<int64_t>(q2))));
  fx_u64 q = (static_cast<fx_u64>(s1) << 27) + static_cast<fx_u64>(static_cast<int64_t>(q2));
  if (rem2 < 0) {
    q -= 1;
    rem2 += static_cast<int64_t>(2 * q + 1);
    if (rem2 < 0) q -= 1;
  } else if (rem2 > static_cast<int64_t>(2 * q)) {
    rem2 -= static_cast<int64_t>(2 * q + 1);
    q += 1;
    if (rem2 > static_cast<int64_t>(2 * q)) q += 1;
  }
  const fx_u64 m = (q + 1) >> 1;
  *s = fx_dbl(m + (static_cast<fx_u64>(static_cast<unsigned>(((ex - 1023 - odd) >> 1) + 1022))
                   << 52));
  return static_cast<unsigned>(ex - 1) < 2046u;
}

// ---- argument reduction -------------------------------------------------------------------------
// |x| * K = n + (fh:fm:fl) / 2^96 for K = c * 2^(1-k), c = (c2:c1:c0) / 2^96 in [1/2, 1), and
// t = exponent(x) + 1 + k in [-32, 31]: the 96-bit product of the mantissa and c, shifted.
struct FxReduced {
  fx_u32 n, fh, fm, fl;
};
CGB_FX FxReduced fx_reduce(fx_u64 b, int t, fx_u32 c2, fx_u32 c1, fx_u32 c0) {
  const fx_u64 m = ((b & kFxMant) | kFxOne) << 11;
  const fx_u32 m1 = static_cast<fx_u32>(m >> 32), m0 = static_cast<fx_u32>(m);
  const fx_u64 t1 = static_cast<fx_u64>(m1) * c0 + fx_mulhi32(m0, c0);
  const fx_u64 t2 = static_cast<fx_u64>(m0) * c1 + static_cast<fx_u32>(t1);
  const fx_u64 t3 = static_cast<fx_u64>(m1) * c1 + (t1 >> 32) + (t2 >> 32);
  const fx_u64 t4 = static_cast<fx_u64>(m0) * c2 + static_cast<fx_u32>(t3);
  const fx_u64 t5 = static_cast<fx_u64>(m1) * c2 + (t3 >> 32) + (t4 >> 32);
  const fx_u32 p4 = static_cast<fx_u32>(t5 >> 32), p3 = static_cast<fx_u32>(t5);
  const fx_u32 p2 = static_cast<fx_u32>(t4), p1 = static_cast<fx_u32>(t2);
  const bool neg = t < 0;
  const fx_u32 a = neg ? 0u : p4, bb = neg ? p4 : p3, c = neg ? p3 : p2, d = neg ? p2 : p1;
  const int s = t & 31;
  FxReduced r;
  r.n = fx_shf(a, 0u, s);
  r.fh = fx_shf(bb, a, s);
  r.fm = fx_shf(c, bb, s);
  r.fl = fx_shf(d, c, s);
  return r;
}

// ---- sin and cos --------------------------------------------------------------------------------
// sin(x) and cos(x) for |x| < 2^15; false outside, and for the few arguments within
// about 2^-24 of a multiple of pi/2 other than 0, whose reduced argument has too few bits here.
CGB_FX bool fx_sincos(double x, double* s, double* c) {
  const fx_u64 b = fx_bits(x);
  const int e = fx_expo(b) - 1023;
  const fx_u64 sx = b & kFxSign;
  if (e < -33) {  // x - x^3/6 rounds to x, zeros and subnormals included
    *s = x;
    *c = 1.0;
    return true;
  }
  if (e > 14) return false;
  const int t = e + 1;
  FxReduced r = fx_reduce(b, t, 0xa2f9836eu, 0x4e441529u, 0xfc2757d1u);  // 2/pi
  // nearest quadrant; |f| <= 1/2 of a quadrant, on the other side when rounded up
  const fx_u32 up = static_cast<fx_u32>(static_cast<int>(r.fh) >> 31);
  const fx_u32 quad = r.n - up;
  r.fh ^= up;
  r.fm ^= up;
  r.fl ^= up;
  const fx_u64 f = (static_cast<fx_u64>(r.fh) << 32) | r.fm;  // Q64
  const fx_u64 z = fx_mulhi(f, f);
  const fx_u32 zh = static_cast<fx_u32>(z >> 32);
  // sin(pi/2 f) / f in z = f^2 (Q63; the last three terms Q50), 1 - cos(pi/2 f) over z
  const fx_u32 s5 = 0xf183a5a8u - fx_mulhi32(zh, 0x3d1dda2u - fx_mulhi32(zh, 0xb62dcu));
  fx_u64 ps = 0x541e0d2172f61ull - fx_mulhi(z, static_cast<fx_u64>(s5) << 13);
  ps = 0x99696673156112ull - fx_mulhi(z, ps);
  ps = 0xa335e33bad56c90ull - fx_mulhi(z, ps);
  ps = 0x52aef39896f94aedull - fx_mulhi(z, ps);
  ps = 0xc90fdaa22168c235ull - fx_mulhi(z, ps);
  const fx_u32 c5 = 0xfce7122eu - fx_mulhi32(zh, 0x365e7d6u);
  fx_u64 pc = 0xd368f77a3cdfull - fx_mulhi(z, static_cast<fx_u64>(c5) << 10);
  pc = 0x1e1f5068688d5bull - fx_mulhi(z, pc);
  pc = 0x2aba78fc796481eull - fx_mulhi(z, pc);
  pc = 0x20783e1036b5808aull - fx_mulhi(z, pc);
  pc = 0x9de9e64df22ef2ceull - fx_mulhi(z, pc);
  // cos: 1 - z pc, in [0.7, 1]: Q64 after one doubling of the Q63 product (2^64 itself: 1)
  const fx_u64 cz = fx_mulhi(z, pc) << 1;
  const double cv = cz ? fx_pack(0ull - cz, 1022, 0) : 1.0;
  // sin: f normalised times ps
  const int lz = r.fh ? fx_clz64(f) : 32;
  const fx_u64 fn = r.fh ? (f << lz) | (static_cast<fx_u64>(r.fl) >> (32 - (lz & 31)))
                         : (static_cast<fx_u64>(r.fm) << 32) | r.fl;
  const int lz2 = r.fh ? 0 : fx_clz64(fn);
  fx_u64 sv = fx_mulhi(fn << lz2, ps);  // in (2^62, 2^63.7)
  const int one = static_cast<int>(sv >> 63) ^ 1;
  sv <<= one;
  const double sn = fx_pack(sv, 1023 - lz - lz2 - one, 0);
  // quadrants: sin(q + f), cos(q + f) with f's sign folded in
  const fx_u64 fs = up ? kFxSign : 0ull;
  const fx_u64 q0 = (quad & 1u) ? fx_bits(cv) : fx_bits(sn) | fs;
  const fx_u64 q1 = (quad & 1u) ? fx_bits(sn) | fs : fx_bits(cv);
  *s = fx_dbl(q0 ^ sx ^ ((quad & 2u) ? kFxSign : 0ull));
  *c = fx_dbl(q1 ^ (((quad + 1u) & 2u) ? kFxSign : 0ull));
  return t <= 0 || r.fh >= 256u;
}

// ---- exp ----------------------------------------------------------------------------------------
// 2^f for f (Q64) in [0, 1): Q62
CGB_FX fx_u64 fx_exp2(fx_u64 f) {
  const fx_u32 fh = static_cast<fx_u32>(f >> 32);
  const fx_u32 p10 = 0xe0aa3586u + fx_mulhi32(fh, 0x15a6d6bau);
  fx_u64 p = 0x6e257eac0cull + fx_mulhi(f, static_cast<fx_u64>(p10) << 3);
  p = 0x58a2a6c9985ull + fx_mulhi(f, p);
  p = 0x3ffa084011c7ull + fx_mulhi(f, p);
  p = 0x28611ebea3b70ull + fx_mulhi(f, p);
  p = 0x15d87ff7b78a76ull + fx_mulhi(f, p);
  p = 0x9d955b7af7c829ull + fx_mulhi(f, p);
  p = 0x38d611ae0e0109dull + fx_mulhi(f, p);
  p = 0xf5fdeffc15eb3aaull + fx_mulhi(f, p);
  p = 0x2c5c85fdf473f455ull + fx_mulhi(f, p);
  return 0x3fffffffffffffedull + fx_mulhi(f, p);
}
// exp(x) for |x| < 700
CGB_FX bool fx_exp(double x, double* y) {
  const fx_u64 b = fx_bits(x);
  const int e = fx_expo(b) - 1023;
  if (e < -34) {  // 1 + x + x^2/2 rounds as 1 + x
    *y = 1.0 + (e >= -54 ? x : 0.0);
    return true;
  }
  if (e > 9 || (b & ~kFxSign) >= 0x4085e00000000000ull) return false;
  const FxReduced r = fx_reduce(b, e + 2, 0xb8aa3b29u, 0x5c17f0bbu, 0xbe87fed0u);  // log2(e)
  const fx_u32 neg = static_cast<fx_u32>(static_cast<int64_t>(b) >> 63);
  const int n = static_cast<int>(r.n ^ neg);
  const fx_u64 f = (static_cast<fx_u64>(r.fh ^ neg) << 32) | (r.fm ^ neg);
  *y = fx_pack(fx_exp2(f) << 1, 1023 + n, 0);
  return true;
}

// ---- log ----------------------------------------------------------------------------------------
// ln(x) for normal positive x: x = 2^e w with w in [sqrt(1/2), sqrt(2)), ln w = s L(s^2) with
// s = (w - 1)/(w + 1) and L(z) = (2/s) atanh(s)
CGB_FX bool fx_log(double x, double* y) {
  const fx_u64 b = fx_bits(x);
  const int ex = static_cast<int>(b >> 52);
  if (static_cast<unsigned>(ex - 1) >= 2046u || b == 0x3ff0000000000000ull) {
    *y = 0.0;
    return b == 0x3ff0000000000000ull;
  }
  const fx_u64 m = (b & kFxMant) | kFxOne;
  const int half = m > 0x16a09e667f3bccull ? 1 : 0;  // sqrt(2)
  const int e = ex - 1023 + half;
  const fx_u64 one = kFxOne << half;
  const fx_u64 num = half ? one - m : m - one;  // w - 1, negative when halved
  const fx_u64 den = (m + one) << 10;           // (w + 1) or (w + 1)/2: Q63 in [1, 2)
  const fx_u64 r = fx_rcp62(den);
  const int lz = fx_clz64(num | 1u);
  const fx_u64 sn = fx_mulhi(num << lz, r);  // s normalised, top bit 62 or 63
  const int sh = lz - 11;
  const fx_u64 sq = sh < 64 ? sn >> sh : 0;  // Q64
  const fx_u64 z = fx_mulhi(sq, sq);
  const fx_u32 l6 = 0x9ccc7ac0u + fx_mulhi32(static_cast<fx_u32>(z >> 32), 0x97aae37au);
  fx_u64 p = 0xba33506cf1a0171ull + fx_mulhi(z, static_cast<fx_u64>(l6) << 28);
  p = 0xe38e27ee660a9ccull + fx_mulhi(z, p);
  p = 0x1249249453e87d3full + fx_mulhi(z, p);
  p = 0x1999999997aba897ull + fx_mulhi(z, p);
  p = 0x2aaaaaaaaaab5c49ull + fx_mulhi(z, p);
  p = 0x7ffffffffffffff6ull + fx_mulhi(z, p);  // Q62 in [2, 2.03)
  fx_u64 v;
  int expo;
  fx_u64 sign;
  if (e == 0) {
    v = fx_mulhi(sn, p);  // ln w = v 2^(-lz - 53 + 2)
    const int nz = fx_clz64(v);
    v <<= nz;
    expo = 1023 + 63 - nz - lz - 51;
    sign = half ? kFxSign : 0;
  } else {
    // |e| ln 2 (Q64, 96 bits) plus or minus ln w
    const fx_u32 ae = static_cast<fx_u32>(e < 0 ? -e : e);
    const fx_u64 lo = static_cast<fx_u64>(ae) * 0xd1cf79acu;
    const fx_u64 hi = static_cast<fx_u64>(ae) * 0xb17217f7u + (lo >> 32);
    fx_u64 f = (hi << 32) | static_cast<fx_u32>(lo);
    fx_u32 i = static_cast<fx_u32>(hi >> 32);
    const fx_u64 w = fx_mulhi(sq, p) << 2;
    if ((half != 0) == (e < 0)) {
      f += w;
      i += f < w;
    } else {
      i -= f < w;
      f -= w;
    }
    // i:f normalised
    const int li = fx_clz64((static_cast<fx_u64>(i) << 32) | (f >> 32));
    v = li < 32 ? (static_cast<fx_u64>(i) << (32 + li)) | (f >> (32 - li)) : f << (li - 32);
    expo = 1023 + 31 - li;
    sign = e < 0 ? kFxSign : 0;
  }
  *y = fx_pack(v, expo, sign);
  return true;
}

// ---- tanh ---------------------------------------------------------------------------------------
CGB_FX bool fx_tanh(double x, double* y) {
  const fx_u64 b = fx_bits(x);
  const int e = fx_expo(b) - 1023;
  const fx_u64 sx = b & kFxSign;
  if (e == -1023) {  // zeros and subnormals: x - x^3/3 rounds to x
    *y = x;
    return true;
  }
  if (e < -3) {
    // x (1 - z (t1 - z (t2 - ...))), z = x^2 < 2^-6
    const fx_u64 m = ((b & kFxMant) | kFxOne) << 11;
    const int sh = -(e + 1);
    const fx_u64 q = sh < 64 ? m >> sh : 0;
    const fx_u64 z = fx_mulhi(q, q);
    const fx_u32 t5 = 0x913226aeu - fx_mulhi32(static_cast<fx_u32>(z >> 32), 0x39bf9d57u);
    fx_u64 p = 0x5993cf90631d267ull - fx_mulhi(z, static_cast<fx_u64>(t5) << 26);
    p = 0xdd0dd0daa71cb76ull - fx_mulhi(z, p);
    p = 0x222222222214f794ull - fx_mulhi(z, p);
    p = 0x555555555555549aull - fx_mulhi(z, p);
    fx_u64 v = m - fx_mulhi(m, fx_mulhi(z, p));
    const int one = static_cast<int>(v >> 63) ^ 1;
    *y = fx_pack(v << one, e + 1023 - one, sx);
    return true;
  }
  if (e > 4) {  // |x| >= 32: 1 - 2 exp(-64) rounds to 1; NaN goes to the caller
    *y = fx_dbl(sx | 0x3ff0000000000000ull);
    return e < 1024;
  }
  // (1 - t)/(1 + t), t = 2^-v, v = 2 |x| log2(e)
  const FxReduced r = fx_reduce(b, e + 3, 0xb8aa3b29u, 0x5c17f0bbu, 0xbe87fed0u);
  const fx_u64 f = ~((static_cast<fx_u64>(r.fh) << 32) | r.fm);
  fx_u64 t = r.n < 63u ? (fx_exp2(f) << 1) >> r.n : 1u;  // Q64
  t = t ? t : 1u;
  const fx_u64 q = fx_mulhi(0ull - t, fx_rcp62(kFxSign + (t >> 1)));
  const int lz = fx_clz64(q);
  *y = fx_pack(q << lz, 1022 - lz, sx);
  return true;
}

}  // namespace cgb
