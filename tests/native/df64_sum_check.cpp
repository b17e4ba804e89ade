// df64::sum4 of four double-floats against their exact sum (128-bit integers),
// over random magnitudes and cancelling terms.  Prints the largest error as a
// fraction of 2^-53 times the largest term, and how many sums were checked.
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "eph_df64.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t draw() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}
static double unit() { return (double)(draw() >> 11) * 0x1p-53; }

int main() {
  double worst = 0.0;
  const long n = 2000000;
  for (long i = 0; i < n; ++i) {
    df64::df v[4];
    double most = 0.0;
    for (int k = 0; k < 4; ++k) {
      double x = (unit() - 0.5) * std::ldexp(1.0, -(int)(draw() % 40));
      if (k && draw() % 3 == 0) x = -((double)v[k - 1].hi + (double)v[k - 1].lo) * (1.0 + unit() * std::ldexp(1.0, -(int)(draw() % 45)));
      v[k] = df64::from_double(x);
      most = std::fmax(most, std::fabs((double)v[k].hi));
    }
    __int128 exact = 0;  // in units of 2^-120
    for (int k = 0; k < 4; ++k)
      for (float p : {v[k].hi, v[k].lo}) {
        int e;
        const float m = std::frexp(p, &e);  // p = m 2^e
        if (m != 0.0f && e - 24 + 120 >= 0) exact += (__int128)(int64_t)(m * 0x1p24f) << (e - 24 + 120);
      }
    const double s = df64::sum4(v[0], v[1], v[2], v[3]);
    int e;
    const double m = std::frexp(s, &e);
    __int128 got = 0;
    if (m != 0.0) {
      const int64_t w = (int64_t)(m * 0x1p53);
      const int sh = e - 53 + 120;
      got = sh >= 0 ? (__int128)w << sh : (__int128)(w >> -sh);
    }
    const double err = std::fabs((double)(got - exact)) * 0x1p-120;
    worst = std::fmax(worst, err / (0x1p-53 * most));
  }
  std::printf("%.3f %ld\n", worst, n);
}
