// Double-precision operations on the integer and single-precision pipes.
//
// GB300 issues two double-precision lanes per SM and clock (one warp
// instruction every 64 clocks per scheduler) against 64 integer lanes, so a
// double division (about ten dependent FP64 instructions), a square root, a
// comparison, a min / max or an exact scaling by a power of two costs far
// more there than the same result formed with integer instructions.  The
// functions here return what IEEE 754 round-to-nearest arithmetic returns, bit
// for bit; additions and products stay on the FP64 pipe.
//
// Division and square root: two radix-2^28/2^29 quotient (root) digits from a
// 31-bit reciprocal (reciprocal root) estimate, refined by one Newton step
// from the hardware's single-precision approximation, give the result to a few
// units of its 58th bit; the exact sign of the remainder at the midpoint of
// the two candidate results then decides the rounding (a quotient or root of
// 53-bit operands is never a midpoint).  Schoolbook digit recurrence and
// remainder test, as in Knuth, The Art of Computer Programming, vol. 2, 4.3.1,
// and Brent and Zimmermann, Modern Computer Arithmetic, 2.4 and 3.5.
// Division and square root are calls, not inlined: a step has tens of call
// sites, and the smaller kernels run faster at two resident CTAs per SM (3D
// 160^3 step: 8.28 ms against 9.3 ms inlined).
// Subnormal operands and results take a longer integer path; NaN, infinities,
// zero divisors and overflows the hardware operation.
//
// The header also compiles on the host, where a test compares every function
// with the host's IEEE operations.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define TFV_SOFT __device__ __forceinline__
#define TFV_SOFT_CALL static __device__ __noinline__
#else
#include <cmath>
#include <cstring>
#define TFV_SOFT inline
#define TFV_SOFT_CALL inline
#endif

namespace tfv {

#if defined(__CUDACC__)
TFV_SOFT uint32_t s64_hi(double x) { return (uint32_t)__double2hiint(x); }
TFV_SOFT uint32_t s64_lo(double x) { return (uint32_t)__double2loint(x); }
TFV_SOFT double s64_make(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
TFV_SOFT uint32_t s64_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
TFV_SOFT float s64_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
TFV_SOFT float s64_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
TFV_SOFT uint32_t s64_u32(float x) { return __float2uint_rz(x); }
TFV_SOFT int s64_clz(uint64_t x) { return __clzll((long long)x); }
#else
TFV_SOFT uint64_t s64_bits(double x) {
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
}
TFV_SOFT uint32_t s64_hi(double x) { return (uint32_t)(s64_bits(x) >> 32); }
TFV_SOFT uint32_t s64_lo(double x) { return (uint32_t)s64_bits(x); }
TFV_SOFT double s64_make(uint32_t hi, uint32_t lo) {
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}
TFV_SOFT uint32_t s64_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// the host stands in for the approximations with a relative error beyond the
// hardware's (2^-22), of either sign
#ifndef TFV_SOFT_TEST_ERROR
#define TFV_SOFT_TEST_ERROR 0.0f
#endif
TFV_SOFT float s64_rcp(float x) { return (1.0f / x) * (1.0f + (TFV_SOFT_TEST_ERROR)); }
TFV_SOFT float s64_rsqrt(float x) {
  return (1.0f / std::sqrt(x)) * (1.0f + (TFV_SOFT_TEST_ERROR));
}
TFV_SOFT uint32_t s64_u32(float x) { return (uint32_t)x; }
TFV_SOFT int s64_clz(uint64_t x) { return __builtin_clzll(x); }
#endif

TFV_SOFT uint64_t s64_join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// -- quotient ----------------------------------------------------------------
// 2^62 / b32 (31 bits, relative error below 2^-29) for a divisor mantissa B in
// [2^52, 2^53), b32 its leading 32 bits.
TFV_SOFT uint32_t soft_recip62(uint64_t B) {
  const uint32_t b32 = (uint32_t)(B >> 21);
  const uint32_t r0 = s64_u32(s64_rcp((float)b32) * 4611686018427387904.0f);
  const int64_t err = (int64_t)((1ull << 62) - (uint64_t)r0 * b32);
  const uint32_t r = r0 + (uint32_t)(int32_t)(((int64_t)(int32_t)(err >> 16) * (int64_t)(int32_t)(r0 >> 1)) >> 45);
  return r > 0x7fffffffu ? 0x7fffffffu : r;
}
// A 2^57 / B for mantissas with A / B in [1, 2), within 5 units: first digit
// q1 = A 2^29 / B, its exact remainder, second digit.
TFV_SOFT uint64_t soft_quotient57(uint64_t A, uint64_t B, uint32_t r) {
  const uint32_t q1 = s64_mulhi((uint32_t)(A >> 22), r);
  const int64_t rem = (int64_t)((A << 29) - (uint64_t)q1 * B);
  const int32_t q2 = (int32_t)(((int64_t)(int32_t)(rem >> 24) * (int64_t)(int32_t)r) >> 31);
  return ((uint64_t)q1 << 28) + (uint64_t)(int64_t)q2;
}

// a / b where an operand or the result is zero, subnormal or out of range
// (the far field of a blast wave carries subnormal momenta, whose division by
// the hardware sequence is slower still).  Out of line: the common case
// branches around it.
TFV_SOFT_CALL double soft_div_rare(double a, double b) {
  const uint32_t ah = s64_hi(a), al = s64_lo(a), bh = s64_hi(b), bl = s64_lo(b);
  uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  uint64_t A = s64_join(ah & 0xfffffu, al), B = s64_join(bh & 0xfffffu, bl);
  if (ea == 0x7ffu || eb == 0x7ffu || (eb | B) == 0u) return a / b;  // NaN, infinity, x / 0
  if ((ea | A) == 0u) return s64_make(sign, 0u);
  int xa = (int)ea, xb = (int)eb;
  if (ea == 0u) {  // subnormal: normalise
    const int n = s64_clz(A) - 11;
    A <<= n;
    xa = 1 - n;
  } else {
    A |= 1ull << 52;
  }
  if (eb == 0u) {
    const int n = s64_clz(B) - 11;
    B <<= n;
    xb = 1 - n;
  } else {
    B |= 1ull << 52;
  }
  const bool less = A < B;
  A = less ? A << 1 : A;
  const int e = xa - xb + (less ? 1022 : 1023);
  if (e >= 2046) return a / b;  // overflows, or may by rounding
  const uint64_t Q = soft_quotient57(A, B, soft_recip62(B));
  const int drop = e >= 1 ? 5 : 6 - e;  // bits below the result's last one
  if (drop >= 60) return s64_make(sign, 0u);  // below half of the smallest subnormal
  const uint64_t H = ((Q >> drop) << drop) | (1ull << (drop - 1));
  const int64_t gap = (int64_t)(Q - H);
  int64_t side = gap;  // decided by the quotient's estimate ...
  if (gap <= 8 && gap >= -8) side = (int64_t)((A << 57) - H * B);  // ... or exactly
  uint64_t m = Q >> drop;
  m += (side > 0 || (side == 0 && (m & 1u))) ? 1u : 0u;  // ties to even
  const uint64_t bits = (e >= 1 ? (uint64_t)(uint32_t)(e - 1) << 52 : 0ull) + m;
  return s64_make((uint32_t)(bits >> 32) | sign, (uint32_t)bits);
}

// A divisor with its reciprocal estimate: several quotients by one divisor
// (the velocities, sound speed and enthalpy of a face state) form it once.
struct SoftDivisor {
  double b;
  uint32_t r;
};
TFV_SOFT SoftDivisor soft_divisor(double b) {
  SoftDivisor d;
  d.b = b;
  d.r = soft_recip62(s64_join((s64_hi(b) & 0xfffffu) | 0x100000u, s64_lo(b)));
  return d;
}

// a / d.b.  Mantissas A, B in [2^52, 2^53); A doubled where A < B, so that
// A / B lies in [1, 2).
TFV_SOFT_CALL double soft_div(double a, const SoftDivisor d) {
  const uint32_t ah = s64_hi(a), al = s64_lo(a), bh = s64_hi(d.b), bl = s64_lo(d.b);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  const uint64_t B = s64_join((bh & 0xfffffu) | 0x100000u, bl);
  uint64_t A = s64_join((ah & 0xfffffu) | 0x100000u, al);
  const bool less = A < B;
  A = less ? A << 1 : A;
  const int e = (int)ea - (int)eb + (less ? 1022 : 1023);  // biased exponent of a / b
  const uint64_t Q = soft_quotient57(A, B, d.r);
  // midpoint between the candidates (Q >> 5) and (Q >> 5) + 1
  const uint64_t H = (Q & ~31ull) | 16ull;
  const int64_t side = (int64_t)((A << 57) - H * B);
  const uint64_t m = (Q >> 5) + (side > 0 ? 1u : 0u);
  const uint64_t bits = ((uint64_t)(uint32_t)(e - 1) << 52) + m;
  const bool normal = (ea - 1u < 2046u) && (eb - 1u < 2046u) && ((uint32_t)(e - 1) < 2045u);
  if (normal) return s64_make((uint32_t)(bits >> 32) | sign, (uint32_t)bits);
  // zero over a normal number (quiescent gas): a zero with the quotient's sign
  if (((ah << 1) | al) == 0u && eb - 1u < 2046u) return s64_make(sign, 0u);
  return soft_div_rare(a, d.b);
}
TFV_SOFT double soft_div(double a, double b) { return soft_div(a, soft_divisor(b)); }

// -- square root ---------------------------------------------------------------
TFV_SOFT_CALL double soft_sqrt(double x) {
  const uint32_t xh = s64_hi(x), xl = s64_lo(x);
  if (xh - 0x00100000u >= 0x7fe00000u) {  // zero, subnormal, negative, infinite or NaN
#if defined(__CUDACC__)
    return sqrt(x);
#else
    return std::sqrt(x);
#endif
  }
  const uint32_t odd = ((xh >> 20) & 1u) ^ 1u;  // unbiased exponent odd
  const uint32_t er = ((xh >> 20) - 1023u - odd) / 2u;  // exact: an even difference (mod 2^32)
  uint64_t M = s64_join((xh & 0xfffffu) | 0x100000u, xl);
  M = odd ? M << 1 : M;  // [2^52, 2^54)
  // y = 2^46 / sqrt(m32) (30 to 31 bits), m32 the leading 32 bits
  const uint32_t m32 = (uint32_t)(M >> 22);
  const uint32_t y0 = s64_u32(s64_rsqrt((float)m32) * 70368744177664.0f);
  const uint32_t u = (uint32_t)(((uint64_t)y0 * y0) >> 31);
  const int64_t err = (int64_t)((1ull << 61) - (uint64_t)u * m32) * 2;
  uint32_t y = y0 + (uint32_t)(int32_t)(((int64_t)(int32_t)(err >> 16) * (int64_t)(int32_t)(y0 >> 1)) >> 46);
  y = y > 0x7fffffffu ? 0x7fffffffu : y;
  // digits of sqrt(M 2^62)
  const uint32_t s1 = s64_mulhi(m32, y);  // sqrt(M) 2^3
  const int64_t rem = (int64_t)((M << 6) - (uint64_t)s1 * s1);
  const int32_t s2 = (int32_t)(((int64_t)(int32_t)(rem >> 4) * (int64_t)(int32_t)y) >> 29);
  const uint64_t S = ((uint64_t)s1 << 28) + (uint64_t)(int64_t)s2;  // within 12 units
  // midpoint of the candidates, in units of sqrt(M 2^60)
  const uint64_t H = ((S >> 5) << 4) | 8ull;
  const int64_t side = (int64_t)((M << 60) - H * H);
  const uint64_t m = (S >> 5) + (side > 0 ? 1u : 0u);
  const uint64_t bits = ((uint64_t)(er + 1022u) << 52) + m;
  return s64_make((uint32_t)(bits >> 32), (uint32_t)bits);
}

// -- exact scaling by 1/2 and 2 --------------------------------------------------
TFV_SOFT double soft_half(double x) {
  const uint32_t h = s64_hi(x), l = s64_lo(x), mag = h & 0x7fffffffu;
  if (mag - 0x00200000u < 0x7fd00000u) return s64_make(h - 0x00100000u, l);
  if ((mag | l) == 0u) return x;
  return 0.5 * x;
}
TFV_SOFT double soft_twice(double x) {
  const uint32_t h = s64_hi(x), l = s64_lo(x), mag = h & 0x7fffffffu;
  if (mag - 0x00100000u < 0x7fd00000u) return s64_make(h + 0x00100000u, l);
  if ((mag | l) == 0u) return x;
  return 2.0 * x;
}

// -- comparisons -------------------------------------------------------------------
TFV_SOFT bool soft_isnan(double x) {
  const uint32_t mag = s64_hi(x) & 0x7fffffffu;
  return mag > 0x7ff00000u || (mag == 0x7ff00000u && s64_lo(x) != 0u);
}
TFV_SOFT bool soft_isfinite(double x) { return (s64_hi(x) & 0x7fffffffu) < 0x7ff00000u; }
// integer with the order of the (non-NaN) doubles; both zeros map to 0
TFV_SOFT int64_t s64_key(double x) {
  const uint32_t h = s64_hi(x);
  const int64_t s = (int64_t)((int32_t)h >> 31);
  const int64_t mag = (int64_t)s64_join(h & 0x7fffffffu, s64_lo(x));
  return (mag ^ s) - s;
}
TFV_SOFT bool soft_lt(double a, double b) {
  return s64_key(a) < s64_key(b) && !soft_isnan(a) && !soft_isnan(b);
}
TFV_SOFT bool soft_le(double a, double b) {
  return s64_key(a) <= s64_key(b) && !soft_isnan(a) && !soft_isnan(b);
}
// against a positive constant c (compile-time, finite): one 64-bit integer
// comparison, since a negative double is a negative integer
TFV_SOFT bool soft_gt_pos(double x, double c) {
  return (int64_t)s64_join(s64_hi(x), s64_lo(x)) > (int64_t)s64_join(s64_hi(c), s64_lo(c)) &&
         !soft_isnan(x);
}
// x <= 0, x < 0, x > 0, x >= 0 (false for NaN)
TFV_SOFT bool soft_le0(double x) {
  const int64_t k = (int64_t)s64_join(s64_hi(x), s64_lo(x));
  return k <= 0 && !soft_isnan(x);
}
TFV_SOFT bool soft_gt0(double x) {
  const int64_t k = (int64_t)s64_join(s64_hi(x), s64_lo(x));
  return k > 0 && !soft_isnan(x);
}
TFV_SOFT bool soft_lt0(double x) {
  const uint32_t h = s64_hi(x);
  return (int32_t)h < 0 && (((h << 1) | s64_lo(x)) != 0u) && !soft_isnan(x);
}
TFV_SOFT bool soft_ge0(double x) {
  const uint32_t h = s64_hi(x);
  return ((int32_t)h >= 0 || ((h << 1) | s64_lo(x)) == 0u) && !soft_isnan(x);
}
// |x| < c for a positive constant c (false for NaN)
TFV_SOFT bool soft_abs_lt(double x, double c) {
  return s64_join(s64_hi(x) & 0x7fffffffu, s64_lo(x)) < s64_join(s64_hi(c), s64_lo(c));
}

// numpy.maximum / numpy.minimum: NaN propagates, the first operand wins ties
TFV_SOFT double soft_max(double a, double b) {
  const bool first = soft_isnan(a) || (s64_key(a) >= s64_key(b) && !soft_isnan(b));
  return first ? a : b;
}
TFV_SOFT double soft_min(double a, double b) {
  const bool first = soft_isnan(a) || (s64_key(a) <= s64_key(b) && !soft_isnan(b));
  return first ? a : b;
}
// numpy.maximum(x, c) for a positive constant c
TFV_SOFT double soft_max_pos(double x, double c) {
  const bool first =
      (int64_t)s64_join(s64_hi(x), s64_lo(x)) >= (int64_t)s64_join(s64_hi(c), s64_lo(c)) ||
      soft_isnan(x);
  return first ? x : c;
}
// the larger of a running maximum m (>= +0, not NaN) and x; NaN x is ignored,
// as fmax does
TFV_SOFT double soft_fmax_run(double m, double x) {
  const int64_t k = (int64_t)s64_join(s64_hi(x), s64_lo(x));
  const bool take = k > (int64_t)s64_join(s64_hi(m), s64_lo(m)) && !soft_isnan(x);
  return take ? x : m;
}

// -- limiters ------------------------------------------------------------------------
// phi(r) in double precision, region by region: the numpy.maximum /
// numpy.minimum nests of the reference reduce to comparisons of r with
// constants whose low word is zero, decided by r's high word, and each region
// returns the nest's value bit for bit (zeros with their sign; NaN for NaN, but
// 0 in 2D VanLeer and Albada, whose reference selects on r > 0).
template <int DIM, int LIM>
TFV_SOFT double limiter_phi(double r) {
  const uint32_t h = s64_hi(r), l = s64_lo(r);
  const bool nan = soft_isnan(r);
  const bool zero = ((h << 1) | l) == 0u;
  const bool pos = (int32_t)h >= 0 && !zero;  // r > 0 (NaN apart)
  double phi;
  if (LIM == 0) {  // VanLeer: 2 pos / (1 + pos), pos = max(r, 0)
    phi = soft_div(soft_twice(r), 1.0 + r);
    if (!pos) phi = (DIM == 3 && zero) ? r : 0.0;  // max(-0, 0) is -0
  } else if (LIM == 1) {  // Albada: (pos^2 + pos) / (pos^2 + 1)
    const double q = r * r;
    phi = soft_div(q + r, q + 1.0);
    if (!pos) phi = 0.0;
  } else if (LIM == 2) {  // MINBEE: max(0, min(r, 1))
    phi = h < 0x3ff00000u ? r : 1.0;
    if (!pos) phi = 0.0;
  } else if (LIM == 3) {  // Superbee: max(0, max(min(2r, 1), min(r, 2)))
    phi = h < 0x40000000u ? r : 2.0;
    if (h < 0x3ff00000u) phi = h < 0x3fe00000u ? soft_twice(r) : 1.0;
    if (!pos) phi = 0.0;
  } else {  // Unos: max(0, min(min(2, 2r), (2 + r) / 3 [, (1 + 2r) / 3 in 3D]))
    const double r2 = soft_twice(r);
    const double m = h >= 0x3ff00000u ? 2.0 : r2;
    const double a = soft_div(2.0 + r, 3.0);
    phi = DIM == 3 ? soft_min(soft_min(m, a), soft_div(1.0 + r2, 3.0)) : soft_min(m, a);
    if (!pos) phi = 0.0;
  }
  return nan ? (DIM == 2 && LIM < 2 ? 0.0 : r) : phi;
}

}  // namespace tfv
