// g5_exact64.h — IEEE double division, reciprocal-shared division and square
// root on the integer pipes, correctly rounded (round to nearest even), for
// the FP64 form of the step.
//
// Why: GB300 issues 1.66 FP64 instructions per clock per SM against 64 to 128
// integer ones, and a hardware division or square root is seven to nine FP64
// instructions (0.23 per clock per SM).  The integer forms below are about 55
// (division), 30 (a further quotient of the same divisor) and 55 (square
// root) integer instructions and leave the FP64 pipe to the additions and
// products.
//
// Method (from the mathematics; no table, no library constant): the operand's
// 53-bit mantissa as an integer, a 24-bit float approximation y0 of 1/b or
// 1/sqrt(m), its exact residual e = 1 - b y0 (or 1 - m y0^2) in integer
// arithmetic modulo 2^64, one third-order correction (y0 (1 + e + e^2), y0 (1
// + e/2 + 3 e^2/8)), and the 63-bit result of one 64x64 multiplication.  Its
// error is a few units of the 63rd bit (bounds at each function), so the
// rounding to 53 bits is certain unless the ten bits below are within that
// error of the midpoint; only then the sign of the exact remainder decides.
// A seed is kept in [1/2, 1), where its mantissa bits are all of it: next to
// either end (a mantissa just below 2 or 4, or at 1) the approximation may step
// over.
// A quotient or root of doubles is never exactly a midpoint.
//
// Range.  Operands are zero or normal (never subnormal, infinite or NaN); a
// result outside 2^-900 .. 2^700 (zero aside) sets `bad` and the caller
// evaluates its expression with the hardware operations.  With values from
// memory tested once (x64_raw_bad) the operands need no test of their own:
// every value is then a multiple of 2^-954 and so are all sums, which are
// therefore zero or normal, and no sum comes near the overflow.  The functions
// compile for the host too, where the CPU tests compare them with the host's
// operations.
#pragma once

#include <cstdint>
#include <cstring>
#if !defined(__CUDA_ARCH__)
#include <cmath>
#endif

#if defined(__CUDACC__)
#define G5_HD __host__ __device__ __forceinline__
#else
#define G5_HD inline
#endif

namespace g5
{

G5_HD uint32_t
x64_hi(double x)
{
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32);
#endif
}

G5_HD uint32_t
x64_lo(double x)
{
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return (uint32_t)b;
#endif
}

G5_HD double
x64_make(uint32_t hi, uint32_t lo)
{
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double         x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// whether a value from memory is neither zero nor within 2^-900 .. 2^700
G5_HD bool
x64_raw_bad(double x)
{
  const uint32_t h = x64_hi(x) << 1;
  return h - (123u << 21) >= (1600u << 21) && (h | x64_lo(x)) != 0u;
}

// whether an exponent field less one, in place (what the mantissa's leading
// bit completes), leaves 2^-900 .. 2^700
G5_HD bool
x64_range_bad(uint32_t t)
{
  return t - (122u << 20) >= (1601u << 20);
}

// the mantissa as a 63-bit integer, its leading bit at 62
G5_HD uint64_t
x64_mant(uint32_t hi, uint32_t lo)
{
  return ((uint64_t)((hi & 0x000FFFFFu) | 0x00100000u) << 42) | ((uint64_t)lo << 10);
}

// bits of a float approximation of 1/f (f in [1, 2]) within 2^-23, of
// 1/sqrt(f) (f in [1, 4]) within 2^-22.9 of its value, which is what PTX
// promises for the two instructions; f by its bits
G5_HD uint32_t
x64_seed_rcp(uint32_t fb)
{
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &fb, 4);
  f = 1.0f / f;
  std::memcpy(&fb, &f, 4);
  return fb;
#endif
}

G5_HD uint32_t
x64_seed_rsqrt(uint32_t fb)
{
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &fb, 4);
  f = 1.0f / std::sqrt(f);
  std::memcpy(&fb, &f, 4);
  return fb;
#endif
}

// a mantissa (of 20 and 32 bits) rounded to 24 bits, as the bits of a float in
// [1, 2], of one in [2, 4] with `odd`
G5_HD uint32_t
x64_float_mant(uint32_t hi, uint32_t lo, uint32_t odd)
{
  return 0x3F800000u + (odd << 23) + (((hi & 0x000FFFFFu) << 3) | (lo >> 29)) + ((lo >> 28) & 1u);
}

// a seed as an integer multiple of 2^-24, in [2^23, 2^24)
G5_HD uint32_t
x64_seed_mant(uint32_t sb)
{
  sb = sb > 0x3F7FFFFFu ? 0x3F7FFFFFu : sb;
  sb = sb < 0x3F000000u ? 0x3F000000u : sb;
  return (sb & 0x007FFFFFu) | 0x00800000u;
}

G5_HD uint64_t
x64_mulhi3(uint64_t a, uint64_t b)
{
  // the high 64 bits of a b without the low x low product and with the two
  // middle products truncated: 0 to 3 below the exact value
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
}

// whether the top 53 of 63 bits (bit 62 set) need the exact remainder: the
// ten bits below are within 8 units of the midpoint
G5_HD bool
x64_near_half(uint64_t q)
{
  return (((uint32_t)q + (8u - 0x200u)) & 0x3FFu) <= 16u;
}

// A divisor's reciprocal, shared by its quotients.
struct Recip64
{
  uint64_t y;      // 2^64 / (mantissa in [1, 2)), within 2 units
  uint32_t hi, lo; // the divisor
};

// y0 = m 2^-24 from the float seed (of x64_float_mant's bits): |e| < 2^-21.6
// (2^-23 from the seed and 2^-24 from rounding the mantissa to 24 bits, times
// the mantissa).  y0 (1 + e + e^2) is e^3 < 2^-64.8 away, half a unit of y; D
// is exact, the truncations of T weigh 2^-12 units of y, the two shifts of z
// at most one unit.
G5_HD Recip64
recip64_seeded(double b, uint32_t seed, bool & bad)
{
  Recip64 r;
  r.hi = x64_hi(b);
  r.lo = x64_lo(b);
  bad = bad || (r.hi & 0x7FF00000u) == 0u; // a zero divisor
  const uint32_t mh = (r.hi & 0x000FFFFFu) | 0x00100000u;
  const uint32_t m = x64_seed_mant(seed);
  // D = 2^76 e, exact modulo 2^64, |D| < 2^54.4
  const int64_t D = (int64_t)(0u - ((uint64_t)m * r.lo + ((uint64_t)(m * mh) << 32)));
  // T = 2^76 (e + e^2)
  const int32_t Dh = (int32_t)(D >> 24);
  const int64_t T = D + (((int64_t)Dh * Dh) >> 28);
  // y = m 2^40 (1 + T / 2^76)
  const int64_t z = (int64_t)(int32_t)m * (int32_t)(T >> 32) + (int64_t)(((uint64_t)m * (uint32_t)T) >> 32);
  r.y = ((uint64_t)m << 40) + (uint64_t)(z >> 4);
  return r;
}

G5_HD Recip64
recip64(double b, bool & bad)
{
  return recip64_seeded(b, x64_seed_rcp(x64_float_mant(x64_hi(b), x64_lo(b), 0u)), bad);
}

// a / b.  q holds the quotient's top 63 bits to -8 .. +2 units (a y to -4
// .. +1, doubled when the quotient of the mantissas is below 1).
G5_HD double
quot64(double a, const Recip64 & r, bool & bad)
{
  const uint32_t ha = x64_hi(a), la = x64_lo(a), ea = ha & 0x7FF00000u;
  uint64_t       q = x64_mulhi3(x64_mant(ha, la), r.y);
  const bool     small = (uint32_t)(q >> 32) < 0x40000000u;
  q = small ? q + q : q;
  uint64_t M = (q + 0x200u) >> 10;
  if (x64_near_half(q))
  {
    const uint64_t h = 2u * (q >> 10) + 1u; // the midpoint
    const uint64_t b53 = x64_mant(r.hi, r.lo) >> 10;
    M = (q >> 10) + ((int64_t)((x64_mant(ha, la) << (small ? 44 : 43)) - h * b53) > 0 ? 1u : 0u);
  }
  const uint32_t t = ea - (r.hi & 0x7FF00000u) + (small ? 0x3FD00000u : 0x3FE00000u);
  const bool     zero = ea == 0u;
  bad = bad || (!zero && x64_range_bad(t));
  const uint32_t sign = (ha ^ r.hi) & 0x80000000u;
  const uint32_t hi = ((uint32_t)(M >> 32) + t) | sign;
  return x64_make(zero ? sign : hi, zero ? 0u : (uint32_t)M);
}

G5_HD double
div64(double a, double b, bool & bad)
{
  return quot64(a, recip64(b, bad), bad);
}

// whether the root of a high word takes the doubled mantissa
G5_HD uint32_t
x64_odd(uint32_t hi)
{
  return ((hi >> 20) & 1u) ^ 1u;
}

// sqrt(x), x >= 0.  With x = m 4^k, m in [1, 4): N = 2^62 m; y0 = c 2^-24
// from the float seed, e = 1 - m y0^2, |e| < 2^-21.5 (twice the seed's 2^-22.9,
// 2^-24 from rounding the mantissa to 24 bits); y0 (1 + e/2 + 3 e^2/8) is 5 e^3
// / 16 < 2^-66 away; D drops less than one unit of 2^-78 (a seed 2 units of
// 2^-24 off would take D >> 26 past 31 bits).  The root's 63 bits N y come to
// -5 .. +2 units.
G5_HD double
sqrt64_seeded(double x, uint32_t seed)
{
  const uint32_t hx = x64_hi(x), lx = x64_lo(x);
  const bool     zero = hx == 0u;
  const uint32_t mh = (hx & 0x000FFFFFu) | 0x00100000u;
  const uint32_t odd = x64_odd(hx);
  const uint64_t m53 = ((uint64_t)mh << 32) | lx;
  const uint64_t N = m53 << (10u + odd);
  const uint32_t c = x64_seed_mant(seed);
  // D = 2^78 e, modulo 2^64, |D| < 2^57
  const uint64_t W = (uint64_t)c * c;
  const uint32_t wh = (uint32_t)(W >> 32), wl = (uint32_t)W, nh = (uint32_t)(N >> 32), nl = (uint32_t)N;
  const int64_t  D = (int64_t)(0u - (((uint64_t)(wh * nh) << 32) + (uint64_t)wh * nl + (uint64_t)wl * nh + (((uint64_t)wl * nl) >> 32)));
  // T = 2^78 (e/2 + 3 e^2/8)
  const int32_t Dh = (int32_t)(D >> 26);
  const int64_t T = (D >> 1) + 3 * (((int64_t)Dh * Dh) >> 29);
  const int64_t z = (int64_t)(int32_t)c * (int32_t)(T >> 32) + (int64_t)(((uint64_t)c * (uint32_t)T) >> 32);
  const uint64_t s = x64_mulhi3(N, ((uint64_t)c << 40) + (uint64_t)(z >> 6));
  uint64_t       M = (s + 0x200u) >> 10;
  if (x64_near_half(s))
  {
    const uint64_t h = 2u * (s >> 10) + 1u;
    M = (s >> 10) + ((int64_t)((m53 << (54u + odd)) - h * h) > 0 ? 1u : 0u);
  }
  const uint32_t t = ((((hx >> 20) + 1021u - odd) >> 1) << 20);
  return x64_make(zero ? hx : (uint32_t)(M >> 32) + t, zero ? lx : (uint32_t)M);
}

G5_HD double
sqrt64(double x, bool & bad)
{
  const uint32_t hx = x64_hi(x);
  return sqrt64_seeded(x, x64_seed_rsqrt(x64_float_mant(hx, x64_lo(x), x64_odd(hx))));
}

// a b, correctly rounded (ties to even): the 126-bit product of the 63-bit
// mantissas (ten low zeros each) in four 32x32 products, its lower part kept
// as one sticky bit.  About 40 integer instructions.
G5_HD double
mul64(double a, double b, bool & bad)
{
  const uint32_t ha = x64_hi(a), hb = x64_hi(b);
  const uint32_t ea = ha & 0x7FF00000u, eb = hb & 0x7FF00000u;
  const uint64_t A = x64_mant(ha, x64_lo(a)), B = x64_mant(hb, x64_lo(b));
  const uint32_t Ah = (uint32_t)(A >> 32), Al = (uint32_t)A, Bh = (uint32_t)(B >> 32), Bl = (uint32_t)B;
  const uint64_t p0 = (uint64_t)Al * Bl;
  const uint64_t p1 = (uint64_t)Ah * Bl + (p0 >> 32);
  const uint64_t p2 = (uint64_t)Al * Bh + (uint32_t)p1;
  uint64_t       R = (uint64_t)Ah * Bh + (p1 >> 32) + (p2 >> 32); // [2^60, 2^62)
  R |= ((uint32_t)p2 | (uint32_t)p0) != 0u ? 1u : 0u;
  const bool small = (uint32_t)(R >> 32) < 0x20000000u;
  R = small ? R + R : R;
  const uint64_t M = (R + 0xFFu + (((uint32_t)R >> 9) & 1u)) >> 9;
  const uint32_t t = ea + eb - (small ? 0x40000000u : 0x3FF00000u);
  const bool     zero = ea == 0u || eb == 0u;
  bad = bad || (!zero && x64_range_bad(t));
  const uint32_t sign = (ha ^ hb) & 0x80000000u;
  return x64_make(zero ? sign : ((uint32_t)(M >> 32) + t) | sign, zero ? 0u : (uint32_t)M);
}

} // namespace g5
