// FP64 products and quotients on the integer units, correctly rounded (round
// to nearest, ties to even): the bits of a * b and a / b.
//
// GB300 has two FP64 lanes per SM, so a warp's FP64 instruction takes 16
// cycles of the SM and a division about ten of them, while the integer units
// take a warp instruction per cycle or two and SM quarter.  The bit-for-bit
// (EXACT) sweeps and grid substeps are bound by FP64 issue and latency with
// every other unit idle; a quotient here is some 38 integer instructions, what
// quotients by one divisor share another 35, and a product 36, which pays
// beside FP64 work that fills that pipe.
//
// The mathematics is that of integers: with the 53-bit significands A and B,
// a product is A B rounded at its 53rd bit, and
// the quotient is floor(2^52 A / B) (A doubled first where A < B) from an
// under-estimate Y <= 2^116 / B of the reciprocal (two Newton steps in fixed
// point from the FP32 reciprocal, each below 1 / B whatever the sign of the
// error before it), corrected and rounded by its exact remainder.  No tie
// occurs: a quotient of 53-bit integers is never the middle of two 53-bit
// numbers.  Operands with a biased exponent outside SOFT_LO .. SOFT_HI
// (subnormals, infinities, NaN and results near the ends of the range) take
// the hardware's operation; a zero divided is answered as it is, with the sign
// of the quotient.
#pragma once

#include <cstring>

#ifdef __CUDACC__
#define EPH_SOFT __host__ __device__ __forceinline__
#else
#include <cmath>
#define EPH_SOFT inline
#endif

namespace ephgb {
namespace soft {

typedef unsigned long long u64;
typedef long long s64;

constexpr u64 SIGN = 0x8000000000000000ull;
// biased exponents handled here: those of 2^-510 .. 2^510
constexpr unsigned SOFT_LO = 513u, SOFT_HI = 1533u;

EPH_SOFT u64 bits(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  u64 u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
EPH_SOFT double from_bits(u64 u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((s64)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
EPH_SOFT u64 mulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
EPH_SOFT unsigned exponent(u64 u) { return (unsigned)(u >> 52) & 0x7ffu; }
EPH_SOFT bool in_range(unsigned e) { return e - SOFT_LO <= SOFT_HI - SOFT_LO; }
EPH_SOFT u64 significand(u64 u) { return (u & 0xfffffffffffffull) | 0x10000000000000ull; }

// the hardware's operations, out of line: predicated in place they would take
// the FP64 pipe's cycles whether any lane needs them or not
#ifdef __CUDACC__
#define EPH_SOFT_RARE static __host__ __device__ __noinline__
#else
#define EPH_SOFT_RARE inline
#endif
EPH_SOFT_RARE double hard_mul(double a, double b) { return a * b; }
EPH_SOFT_RARE double hard_div(double a, double b) { return a / b; }

// a * b
EPH_SOFT double mul(double a, double b) {
  const u64 ua = bits(a), ub = bits(b);
  const unsigned ea = exponent(ua), eb = exponent(ub);
  if (!(in_range(ea) && in_range(eb))) return hard_mul(a, b);
  // A 2^11 B: 116 or 117 bits, the upper 64-bit word holding 52 or 53 of them
  const u64 A = significand(ua) << 11, B = significand(ub);
  u64 hi = mulhi(A, B), lo = A * B;
  const unsigned full = (unsigned)(hi >> 52);  // 1: 53 bits
  if (!full) {
    hi = (hi << 1) | (lo >> 63);
    lo <<= 1;
  }
  hi += lo + (hi & 1) > 0x8000000000000000ull ? 1 : 0;  // up above the half, at it to even
  return from_bits(((ua ^ ub) & SIGN) | (hi + ((u64)(ea + eb - 1024u + full) << 52)));
}

// what the quotients by one divisor share
struct Divisor {
  double b;
  u64 B, Y;       // significand; under-estimate of 2^116 / B
  unsigned e;     // biased exponent, 0 where the hardware divides
};

EPH_SOFT Divisor divisor(double b) {
  Divisor d;
  const u64 ub = bits(b);
  d.b = b;
  d.e = exponent(ub);
  if (!in_range(d.e)) d.e = 0;
  d.B = significand(ub);
  const u64 Bn = d.B << 11;  // 2^63 beta, beta in [1, 2)
  // y0 <= 1 from the upper 24 bits, within 4.3e-7 of 1 / beta (truncation and
  // reciprocal 2^-23 each, the factor that keeps it below 1, one rounding)
  const unsigned top = (unsigned)(Bn >> 40) & 0x7fffffu;
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | top)));
  y *= 0.99999976f;
  const unsigned yb = __float_as_uint(y);
#else
  unsigned fb = 0x3f800000u | top, yb;
  float f;
  std::memcpy(&f, &fb, 4);
  f = (1.0f / f) * 0.99999976f;
  std::memcpy(&yb, &f, 4);
#endif
  // y in [1/2, 1) as a fraction of 2^32
  const unsigned y0 = ((yb & 0x7fffffu) | 0x800000u) << (8 - (126 - (int)(yb >> 23)));
  // Newton: y1 = y0 + y0 (1 - beta y0); the residual as a fraction of 2^63
  const u64 t0 = (Bn >> 32) * (u64)y0 + (((Bn & 0xffffffffull) * (u64)y0) >> 32);
  const int e0 = (int)((s64)(0x7fffffffffffffffull - t0) >> 12);
  const u64 y1 = ((u64)y0 << 32) + (u64)(((s64)y0 * e0) >> 19);
  const int e1 = (int)(s64)(0x7fffffffffffffffull - mulhi(Bn, y1));
  d.Y = y1 + (u64)(((s64)(y1 >> 32) * e1) >> 31);
  return d;
}

// a / d.b
EPH_SOFT double div(double a, const Divisor &d) {
  const u64 ua = bits(a), ub = bits(d.b);
  const unsigned ea = exponent(ua);
  // 1023 - 510 .. 1023 + 510 both ways: the quotient's exponent is in range too
  if (!(in_range(ea) && d.e)) return d.e && (ua << 1) == 0 ? from_bits((ua ^ ub) & SIGN) : hard_div(a, d.b);
  u64 A = significand(ua);
  const unsigned less = A < d.B ? 1u : 0u;
  A <<= less;
  u64 q = mulhi(A, d.Y);  // floor(2^52 A / B) or one less
  const u64 twice = ((A << 52) - q * d.B) << 1;  // 2 x remainder, < 4 B
  q += (twice > d.B ? 1u : 0u) + (twice > 3 * d.B ? 1u : 0u);
  return from_bits(((ua ^ ub) & SIGN) | (q + ((u64)(ea - d.e + 1022u - less) << 52)));
}

}  // namespace soft
}  // namespace ephgb
