// photic_softfp.cuh -- IEEE double division, square root and comparisons on
// the integer and single-precision pipes.
//
// On GB300 one FP64 warp instruction takes 19 clocks of an SM whatever the
// number of live lanes (64 of its quarter: two lanes a clock per SM), a
// comparison as much as an fma, against 0.25-0.33 for an FP32 or integer
// one.  Measured there, eight warps on an SM: a compiled double division
// 144 clocks, a square root 144, a comparison with its select 19.  The
// routines below give the same bits with no FP64 instruction in about
// sixty integer and FP32 ones.
//
//  * div, sqrt -- a single-precision estimate of the quotient (root) in two
//    steps, held as an integer of 42 bits; its exact remainder by modular
//    64-bit arithmetic; eleven more bits from the remainder; the exact final
//    remainder then decides the rounding, so the result is the correctly
//    rounded one whatever the estimates' last bits are (the error of the
//    hardware's reciprocal and reciprocal square root only has to stay
//    below 2^-21).  The shape is that of P. Markstein's and of M. Cornea,
//    J. Harrison and P. T. P. Tang's schemes (Scientific Computing on
//    Itanium-based Systems, 2002): approximate, take the exact remainder,
//    correct.  Zero, subnormal, infinite, NaN and (square root) negative
//    operands, and quotients whose exponent leaves the middle of the range,
//    take the compiled operation.
//  * lt, le -- comparisons of doubles on their bits.
//
// The header compiles for the host too (g++), so the CPU test runs the very
// code the kernels run.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "photic_fastmath.cuh"

#if defined(__CUDACC__)
#define PHOTIC_SF_NOINLINE static __host__ __device__ __noinline__
#else
#define PHOTIC_SF_NOINLINE inline
#endif

namespace photic {
namespace sf {

using fm::bits;
using fm::from_bits;

PHOTIC_FM_HD float f_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, sizeof f);
  return f;
#endif
}
PHOTIC_FM_HD uint32_t u_bits(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, sizeof u);
  return u;
#endif
}
PHOTIC_FM_HD float f_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}
// 1 / x and 1 / sqrt(x) to about 22 bits for x in [1, 4).
PHOTIC_FM_HD float f_rcp(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#elif defined(PHOTIC_SF_PERTURB)
  return PHOTIC_SF_PERTURB(1.0f / x);
#else
  return 1.0f / x;
#endif
}
PHOTIC_FM_HD float f_rsqrt(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#elif defined(PHOTIC_SF_PERTURB)
  return PHOTIC_SF_PERTURB((float)(1.0 / ::sqrt((double)x)));
#else
  return (float)(1.0 / ::sqrt((double)x));
#endif
}

// The rare operands: the compiled operations, out of line.
PHOTIC_SF_NOINLINE double div_rare(double a, double b) { return a / b; }
PHOTIC_SF_NOINLINE double sqrt_rare(double a) { return ::sqrt(a); }

// The significand m in [2^52, 2^53) of a double as two floats: the leading
// 24 bits in [1, 2), and 23 of the other 29 as a value below 2^-23.
PHOTIC_FM_HD void split(uint32_t hi, uint32_t lo, float &fh, float &fl) {
  fh = f_bits((((hi << 3) | (lo >> 29)) & 0x7fffffu) | 0x3f800000u);
  fl = f_bits(((lo >> 6) & 0x7fffffu) | 0x34000000u) - 0x1p-23f;
}

constexpr float kMagic = 12582912.0f;  // 1.5 2^23: rounds to an integer in the low bits
constexpr uint32_t kMagicBits = 0x4b400000u;

// Exponent field within 509 of the bias: a product or a quotient of two such
// doubles is normal.
PHOTIC_FM_HD bool mid(double a) {
  const uint32_t hi = (uint32_t)((uint64_t)bits(a) >> 32);
  return ((hi & 0x7fffffffu) - 0x20000000u) < 0x3fd00000u;
}
PHOTIC_FM_HD bool mid_positive(double a) {
  const uint32_t hi = (uint32_t)((uint64_t)bits(a) >> 32);
  return (hi - 0x20000000u) < 0x3fd00000u;
}
// Exponent within 190 of the bias: chains of a few products stay in mid.
PHOTIC_FM_HD bool near(double a) {
  const uint32_t hi = (uint32_t)((uint64_t)bits(a) >> 32);
  return ((hi & 0x7fffffffu) - 0x34100000u) < 0x17d00000u;
}
PHOTIC_FM_HD bool near_positive(double a) {
  const uint32_t hi = (uint32_t)((uint64_t)bits(a) >> 32);
  return (hi - 0x34100000u) < 0x17d00000u;
}

// a * b, correctly rounded, for normal operands with a normal product: the
// 106-bit product of the significands, its leading 53 bits rounded to
// nearest even.
PHOTIC_FM_HD double mul_mid(double a, double b) {
  const uint64_t ua = (uint64_t)bits(a), ub = (uint64_t)bits(b);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
  const uint32_t bh = (uint32_t)(ub >> 32), bl = (uint32_t)ub;
  const uint32_t Ah = (ah & 0xfffffu) | 0x100000u, Bh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t p0 = (uint64_t)al * bl;
  uint64_t m = (uint64_t)al * Bh + (p0 >> 32);
  m = (uint64_t)Ah * bl + m;
  const uint64_t h = (uint64_t)Ah * Bh + (m >> 32);
  const uint32_t h1 = (uint32_t)(h >> 32), h0 = (uint32_t)h, m0 = (uint32_t)m;
  const uint32_t top = h1 >> 9;  // 1: the product is at least 2 (bit 105)
  const uint32_t k = 20u + top;
  // (h : m0) >> k and the bits below
  const uint64_t q = (((uint64_t)h1 << 32) | h0) << (32u - k);
  uint32_t r0 = (uint32_t)q | (m0 >> k);
  uint32_t r1 = (uint32_t)(q >> 32);
  const uint32_t rest = m0 << (32u - k);
  const uint32_t t = rest | ((uint32_t)p0 != 0u ? 1u : 0u);
  const uint32_t up = t > 0x80000000u - (r0 & 1u) ? 1u : 0u;
  const uint32_t e =
      (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - 0x40000000u + ((top + 0u) << 20);
  uint64_t out = ((((uint64_t)r1 << 32) | r0) + up) + ((uint64_t)e << 32);
  out |= (uint64_t)((ah ^ bh) & 0x80000000u) << 32;
  return from_bits((int64_t)out);
}

// a / b, correctly rounded, for operands in mid; y: 1 / (leading 24 bits of
// b's significand) to 22 bits.
PHOTIC_FM_HD double div_mid(double a, double b, float y) {
  const uint64_t ua = (uint64_t)bits(a), ub = (uint64_t)bits(b);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
  const uint32_t bh = (uint32_t)(ub >> 32), bl = (uint32_t)ub;
  const uint32_t Ah = (ah & 0xfffffu) | 0x100000u, Bh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t A = ((uint64_t)Ah << 32) | al, B = ((uint64_t)Bh << 32) | bl;
  const bool c = A < B;  // A / B below 1: doubled, so that q is in [1, 2)
  float af, afl, bf, bfl;
  split(ah, al, af, afl);
  split(bh, bl, bf, bfl);
  const float s = c ? 2.0f : 1.0f;
  af = af * s;
  afl = afl * s;
  float q0 = af * y;
  q0 = fminf(fmaxf(q0, 1.0f), 2.0f);
  // b (q - q0), its two parts each to 24 bits
  const float r = f_fma(-q0, bf, af) + f_fma(-q0, bfl, afl);
  const uint32_t q0i = u_bits(q0) - 0x3f000000u;  // q0 2^23
  const int32_t q1i = (int32_t)(u_bits(f_fma(r * y, 0x1p41f, kMagic)) - kMagicBits);
  const int64_t Q = (int64_t)((uint64_t)q0i << 18) + q1i;  // q 2^41 to two units
  const uint64_t A2 = c ? A + A : A;
  const int64_t R = (int64_t)((A2 << 41) - (uint64_t)Q * B);  // exact: |R| < 2^55
  const int32_t v = (int32_t)(R >> 34);
  const float vf = f_bits(kMagicBits + (uint32_t)v) - kMagic;
  const int32_t q2 = (int32_t)(u_bits(f_fma(vf, y * 0x1p-7f, kMagic)) - kMagicBits);
  const int64_t R2 = (int64_t)(((uint64_t)R << 11) - (uint64_t)(int64_t)q2 * B);
  int64_t F = (int64_t)((uint64_t)Q << 11) + q2;
  // the nearest integer to q 2^52 (a quotient of two doubles is never half
  // way between two doubles)
  const int64_t t = R2 + R2;
  if (t > (int64_t)B) F += 1;
  if (t < -(int64_t)B) F -= 1;
  const uint32_t e = (ah & 0x7ff00000u) - (bh & 0x7ff00000u) + 0x3ff00000u - (c ? 0x100000u : 0u);
  uint64_t out = (uint64_t)F - (1ull << 52) + ((uint64_t)e << 32);
  out |= (uint64_t)((ah ^ bh) & 0x80000000u) << 32;
  return from_bits((int64_t)out);
}

PHOTIC_FM_HD double div_mid(double a, double b) {
  const uint64_t ub = (uint64_t)bits(b);
  float bf, bfl;
  split((uint32_t)(ub >> 32), (uint32_t)ub, bf, bfl);
  return div_mid(a, b, f_rcp(bf));
}

// a / b, correctly rounded.
PHOTIC_FM_HD double div(double a, double b) {
  return mid(a) && mid(b) ? div_mid(a, b) : div_rare(a, b);
}

// sqrt(x), correctly rounded, for x in mid_positive.
PHOTIC_FM_HD double sqrt_mid(double x) {
  const uint64_t u = (uint64_t)bits(x);
  const uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
  const uint32_t odd = (h >> 20) & 1u ? 0u : 1u;  // odd unbiased exponent
  float f, fl;
  split(h, l, f, fl);
  const float s = odd ? 2.0f : 1.0f;
  f = f * s;
  fl = fl * s;
  const uint64_t M = ((((uint64_t)((h & 0xfffffu) | 0x100000u)) << 32) | l) << odd;
  const float y = f_rsqrt(f);
  float s0 = f * y;
  s0 = fminf(fmaxf(s0, 1.0f), 2.0f);
  const float r = f_fma(-s0, s0, f) + fl;
  const uint32_t s0i = u_bits(s0) - 0x3f000000u;
  const int32_t s1i = (int32_t)(u_bits(f_fma(r * y, 0x1p40f, kMagic)) - kMagicBits);
  const int64_t S = (int64_t)((uint64_t)s0i << 18) + s1i;  // sqrt 2^41 to two units
  const int64_t R = (int64_t)((M << 30) - (uint64_t)S * (uint64_t)S);
  const int32_t v = (int32_t)(R >> 23);
  const float vf = f_bits(kMagicBits + (uint32_t)v) - kMagic;
  const int32_t s2 = (int32_t)(u_bits(f_fma(vf, y * 0x1p-8f, kMagic)) - kMagicBits);
  int64_t F = (int64_t)((uint64_t)S << 11) + s2;
  const int64_t Rf = (int64_t)((M << 52) - (uint64_t)F * (uint64_t)F);
  // F is nearest when (F - 1/2)^2 < M 2^52 < (F + 1/2)^2
  if (Rf > F) F += 1;
  else if (Rf <= -F) F -= 1;
  const uint32_t e = (((h >> 20) + 1023u - odd) >> 1) << 20;
  return from_bits((int64_t)((uint64_t)F - (1ull << 52) + ((uint64_t)e << 32)));
}

// sqrt(x), correctly rounded.
PHOTIC_FM_HD double sqrt(double x) { return mid_positive(x) ? sqrt_mid(x) : sqrt_rare(x); }

// a < b.  Of doubles without a sign bit the bits compare as integers (a NaN
// is above every number); a sign bit on either side takes the compiled
// comparison.
PHOTIC_FM_HD bool lt(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return a < b;
  return ia < ib && ib <= 0x7ff0000000000000LL;
}
// a <= b.
PHOTIC_FM_HD bool le(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return a <= b;
  return ia <= ib && ib <= 0x7ff0000000000000LL;
}

// a / 2, exactly, for a normal a of twice the least normal's size or more.
PHOTIC_FM_HD double half_mid(double a) { return from_bits(bits(a) - (1ll << 52)); }

}  // namespace sf
}  // namespace photic
