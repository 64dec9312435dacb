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
PHOTIC_SF_NOINLINE bool lt_rare(double a, double b) { return a < b; }
PHOTIC_SF_NOINLINE bool le_rare(double a, double b) { return a <= b; }

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

// a < b and a <= b.  Of doubles without a sign bit the bits compare as
// integers (a NaN is above every number); a sign bit on either side takes the
// compiled comparison.  The compiler runs that one beside the integer one;
// the _call forms keep it off the FP64 pipe at the price of a branch: faster
// where that pipe is the bound (8 009 temporal stacks 224 -> 207 ms,
// 1024 x 320 scene 316 -> 313), not in the general fit.
PHOTIC_FM_HD bool lt(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return a < b;
  return ia < ib && ib <= 0x7ff0000000000000LL;
}
PHOTIC_FM_HD bool le(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return a <= b;
  return ia <= ib && ib <= 0x7ff0000000000000LL;
}
PHOTIC_FM_HD bool lt_call(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return lt_rare(a, b);
  return ia < ib && ib <= 0x7ff0000000000000LL;
}
PHOTIC_FM_HD bool le_call(double a, double b) {
  const int64_t ia = bits(a), ib = bits(b);
  if ((ia | ib) < 0) return le_rare(a, b);
  return ia <= ib && ib <= 0x7ff0000000000000LL;
}

// Unsigned keys that order as the doubles do, both zeros alike; 0 for a NaN,
// below every number's.
PHOTIC_FM_HD uint64_t order_key(double a) {
  const uint64_t u = (uint64_t)bits(a), sign = 1ull << 63;
  if ((u & ~sign) > 0x7ff0000000000000ull) return 0;
  if (u == sign) return sign;
  return u & sign ? ~u : u | sign;
}

// a + b * c for c in {1/2, 1, 2}: the product is exact (but for half the
// least exponents and twice the largest, which are multiplied on their
// own), so the fused sum rounds as the separate one.
PHOTIC_FM_HD double add_scaled2(double a, double b, float c) {
  const double cd = from_bits(
      (int64_t)(0x3fe00000u + (c > 0.5f ? 0x100000u : 0u) + (c > 1.0f ? 0x100000u : 0u)) << 32);
  const uint32_t e = (uint32_t)((uint64_t)bits(b) >> 52) & 0x7ffu;
  if (e - 2u > 2042u) return a + b * cd;
  return fma(b, cd, a);
}

// a / 2, exactly, for a normal a of twice the least normal's size or more.
PHOTIC_FM_HD double half_mid(double a) { return from_bits(bits(a) - (1ll << 52)); }

PHOTIC_FM_HD uint64_t mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// (v >> s) rounded to nearest, for s in [1, 63]; the value v is the floor of
// never lies half way (see exp_neg).
PHOTIC_FM_HD uint64_t shift_round(uint64_t v, uint32_t s) { return ((v >> (s - 1)) + 1) >> 1; }

// fm::exp_t(x), bit for bit, for x in (-354, 0): `ok` is cleared where this
// cannot tell (the argument's multiple of ln2/64 nearly half way between two,
// a remainder below 2^-40 or of at most 21 significant bits), with the result
// then undefined.
//
// exp_t spends eleven FP64 operations.  Here the multiple n comes from the
// single-precision pipe; the polynomial's three fused multiply-adds
// c1 = r/120 + 1/24, c2 = c1 r + 1/6, c = c2 r + 1/2, whose results lie in
// known binades, are fixed-point products rounded to the grid of the double;
// six FP64 operations remain.  A product of a 53-bit and a
// 53-bit significand that is shifted down by s >= 62 places could only lie
// half way between two grid points with 61 trailing zeros; with fewer than 21
// in r and fewer than 32 in c1 and c2 it never does.
PHOTIC_FM_HD double exp_neg(double x, bool &ok) {
  const double kL1 = 0x1.62e4200000000p-7, kL2 = 0x1.fdf473de6af28p-28;  // as in exp_t
  const float kInvH = 0x1.715476p+6f, kInvL = 0x1.4ae0cp-20f;            // 64 / ln 2
  const uint64_t u = (uint64_t)bits(x);
  const uint32_t h = (uint32_t)(u >> 32) & 0x7fffffffu, l = (uint32_t)u;
  ok = ok && h - 0x3c300000u < 0x40762000u - 0x3c300000u;  // 2^-60 <= |x| < 354
  // |x| as two floats
  const uint32_t fb = ((h << 3) | (l >> 29)) + 0x40000000u;
  const float xh = f_bits(fb);
  const uint32_t fe = (fb & 0x7f800000u) - (23u << 23);
  const float xl = f_bits(((l >> 6) & 0x7fffffu) | fe) - f_bits(fe);
  float t = f_fma(xh, kInvH, kMagic);
  float nf = t - kMagic;
  float fr = f_fma(xh, kInvH, -nf);
  fr = f_fma(xh, kInvL, fr);
  fr = f_fma(xl, kInvH, fr);
  t = fr + kMagic;  // the first rounding of a large product may be off by one
  t = t - kMagic;
  fr = fr - t;
  nf = nf + t;
  ok = ok && fabsf(fr) < 0.5f - 0x1p-18f;
  const int32_t N = (int32_t)(u_bits(nf + kMagic) - kMagicBits);  // -n
  const uint32_t nb = u_bits(nf);
  // N as a double (2^-127 for 0, which leaves x unchanged below)
  const double nd = from_bits(((int64_t)((nb >> 3) + 0x38000000u) << 32) | (uint32_t)(nb << 29));
  double r = fma(nd, kL1, x);
  r = fma(nd, kL2, r);
  const uint64_t ur = (uint64_t)bits(r);
  const uint32_t rh = (uint32_t)(ur >> 32), rl = (uint32_t)ur;
  const int32_t er = 1023 - (int32_t)((rh >> 20) & 0x7ff);  // |r| in [2^-er, 2^(1-er))
  ok = ok && er <= 40 && (rl << 11) != 0;
  const bool neg = (int32_t)rh < 0;
  const uint64_t mr = ((((uint64_t)((rh & 0xfffffu) | 0x100000u)) << 32) | rl) << 11;
  // c1 on the grid 2^-57, c2 on 2^-55, c on 2^-53 (2^-54 below 1/2)
  uint64_t v = shift_round(mulhi(mr, 0x8888888888888800ull), 12 + er);
  const uint64_t c1 = 0x15555555555555ull + (neg ? 0 - v : v);
  v = shift_round(mulhi(mr, c1), 1 + er);
  const uint64_t c2 = 0x15555555555555ull + (neg ? 0 - v : v);
  v = shift_round(mulhi(mr, c2), neg ? er : 1 + er);
  ok = ok && (uint32_t)c1 != 0 && (uint32_t)c2 != 0;
  const double c = from_bits((int64_t)(0x3fe0000000000000ull + (neg ? 0 - v : v)));
  const double p = fma(r * r, c, r);
  const int j = -N & 63;
#if defined(__CUDA_ARCH__)
  const double2 T = __ldg(reinterpret_cast<const double2 *>(fm::kExp2TabDev) + j);
  const double th = T.x, tl = T.y;
#else
  const double th = fm::kExp2TabHost[2 * j], tl = fm::kExp2TabHost[2 * j + 1];
#endif
  const double y = fma(th, p, tl) + th;
  return from_bits(bits(y) + fm::shl52(-N >> 6));
}

PHOTIC_FM_HD int clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

// s rounded to 53 significant bits, nearest even.
PHOTIC_FM_HD int64_t round53(int64_t s) {
  const int32_t h = (int32_t)(s >> 32);
  const int c = clz((uint32_t)(h ^ (h >> 31)));
  const uint32_t k = c < 11 ? 11u - (uint32_t)c : 0u;
  const uint32_t mask = (1u << k) - 1u;
  const uint32_t lo = (uint32_t)s;
  s += (mask >> 1) + ((lo >> k) & mask & 1u);
  return s & ~(int64_t)mask;
}

// ((0 + v[0]) + v[1]) + ... + v[n-1], then minus v[h], each operation rounded
// as in double, v[j] = p[j * stride] for n <= 7: the doubles as integers on
// the finest one's grid, the running sum rounded to 53 bits after every
// step.  False, with nothing done, for a zero, subnormal or special value or
// where the exponents span more than seven (the sum would leave 63 bits).
PHOTIC_FM_HD bool sum_less_one(const double *p, int stride, int n, int h, double &z) {
  uint32_t emin = 0x7ff, emax = 0;
  for (int j = 0; j < n; j++) {
    const uint32_t e = (uint32_t)((uint64_t)bits(p[j * stride]) >> 52) & 0x7ffu;
    emin = e < emin ? e : emin;
    emax = e > emax ? e : emax;
  }
  if (emin < 256u || emax > 1790u || emax - emin > 7u) return false;
  int64_t acc = 0;
  for (int j = 0; j <= n; j++) {
    const uint64_t u = (uint64_t)bits(p[(j < n ? j : h) * stride]);
    const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
    int64_t m = (int64_t)(((u & 0xfffffffffffffull) | 0x10000000000000ull) << (e - emin));
    if (((int64_t)u < 0) != (j == n)) m = -m;
    acc = round53(acc + m);
  }
  const bool neg = acc < 0;
  const uint64_t a = (uint64_t)(neg ? -acc : acc);
  if (a == 0) {
    z = 0.0;
    return true;
  }
  const uint32_t ah = (uint32_t)(a >> 32);
  const int lz = ah ? clz(ah) : 32 + clz((uint32_t)a);
  const uint64_t m = lz >= 11 ? a << (lz - 11) : a >> (11 - lz);  // exact
  const uint64_t e = (uint64_t)emin + (uint64_t)(11 - lz);
  z = from_bits((int64_t)((m - 0x10000000000000ull) + (e << 52) + (neg ? 1ull << 63 : 0)));
  return true;
}

// ((0 + p[0]) + p[stride]) + ..., n terms, each addition rounded as in double,
// for terms that are not negative: the running sum as a significand and an
// exponent, about thirty integer instructions an addition against one FP64
// instruction, for the ordered sums that one lane of a warp forms where the
// FP64 pipe is the bound.  Subnormal, infinite and NaN terms and negative ones
// are added in double.
PHOTIC_FM_HD double sum_positive(const double *p, int stride, int n) {
  uint64_t m = 0;  // significand, leading bit 61, nine bits of room below
  int32_t ez = 0;
  bool plain = true;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int i = 0; i < n; i++) {
    const uint64_t u = (uint64_t)bits(p[i * stride]);
    const uint32_t h = (uint32_t)(u >> 32);
    const int32_t e = (int32_t)(h >> 20);  // sign and exponent
    const uint64_t t = (((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | (uint32_t)u) << 9;
    if (u == 0) continue;
    plain = plain && (uint32_t)(e - 1) < 0x7feu;
    // the larger exponent's term stays (equal ones in either order)
    const bool swap = e > ez;
    const uint64_t a = swap ? t : m;
    const uint64_t b = swap ? m : t;
    int32_t d = swap ? e - ez : ez - e;
    ez = swap ? e : ez;
    d = d > 63 ? 63 : d;
    const uint64_t c = b >> d;
    const uint64_t s = (a + c) | ((c << d) != b ? 1u : 0u);
    const uint32_t k = (uint32_t)(s >> 62);  // carry
    uint64_t r = s + ((0x100ull << k) - 1u) + ((s >> (9 + k)) & 1u);
    r >>= 9 + k;
    const uint32_t o = (uint32_t)(r >> 53);  // rounded up to the next power
    m = (r >> o) << 9;
    ez += (int32_t)(k + o);
  }
  if (!plain || ez >= 0x7ff) {
    double z = 0.0;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int i = 0; i < n; i++) z = z + p[i * stride];
    return z;
  }
  if (m == 0) return 0.0;
  return from_bits((int64_t)((m >> 9) - (1ull << 52) + ((uint64_t)ez << 52)));
}

}  // namespace sf
}  // namespace photic
