// df64::sqrt_near as the EAM force sweep uses it, against long double: prints the
// largest relative error in units of 2^-47 over estimates y off by up to 2^-22.
#include <cstdint>
#include <cstdio>

#include "eph_df64.cuh"

static uint64_t state = 88172645463325252ull;
static double unit() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return (double)(state >> 11) / 9007199254740992.0;
}

int main() {
  long double worst = 0.0L;
  for (long i = 0; i < 4000000; ++i) {
    const df64::df a = df64::from_double(std::ldexp(1.0 + 3.0 * unit(), 2 * (int)(i % 20) - 20));
    const float y = (float)((1.0 + (2.0 * unit() - 1.0) * 2.384e-7) / std::sqrt((double)a.hi));
    const df64::df r = df64::sqrt_near(a, df64::mul(a, df64::rsqrt(a, y)), y);
    const long double root = sqrtl((long double)a.hi + a.lo);
    worst = fmaxl(worst, fabsl((long double)r.hi + r.lo - root) / root);
  }
  std::printf("%.3f\n", (double)(worst * 140737488355328.0L));
}
