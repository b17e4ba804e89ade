// Products and quotients of eph_softfp.cuh against the processor's, bit by
// bit, over operands drawn to hit their edges: long runs of zeros and ones in
// the significands, nearly equal significands, exponents on both sides of the
// handled range, zeros, subnormals, infinities.  Prints the number of
// differences per operation.
#include <cstdio>

#include "eph_softfp.cuh"

using namespace ephgb::soft;

static u64 state = 88172645463325252ull;
static u64 draw() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}

static u64 operand(bool any_exponent) {
  u64 m = draw() & 0xfffffffffffffull;
  switch (draw() % 8) {
    case 0: m &= 0xff; break;
    case 1: m |= 0xfffffffffff00ull; break;
    case 2: m &= ~0ull << (draw() % 52); break;
    case 3: m |= (1ull << (draw() % 52)) - 1; break;
  }
  u64 e = any_exponent ? draw() % 2048 : 900 + draw() % 250;
  if (!any_exponent && draw() % 4 == 0) e = (draw() & 1) ? 511 + draw() % 5 : 1531 + draw() % 5;
  if (draw() % 64 == 0) e = m = 0;
  return (draw() << 63) | (e << 52) | (m & 0xfffffffffffffull);
}

static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }

int main() {
  long bad_mul = 0, bad_div = 0;
  for (long i = 0; i < 20000000; ++i) {
    const u64 a = operand(i % 16 == 0);
    u64 b = operand(i % 16 == 0);
    if (i % 7 == 0) b = (b & ~0xfffffffffffffull) | ((a + draw() % 9 - 4) & 0xfffffffffffffull);
    const double x = from_bits(a), y = from_bits(b);
    bad_mul += !same(mul(x, y), x * y);
    bad_div += !same(div(x, divisor(y)), x / y);
  }
  std::printf("mul %ld\ndiv %ld\n", bad_mul, bad_div);
}
