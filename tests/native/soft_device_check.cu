// The device half of eph_softfp.cuh: quotients and products against the
// hardware's, bit by bit.  Every one of the 2^23 leading divisor significands,
// which choose the approximate reciprocal the quotient starts from, with the
// rest of the divisor's bits all zero, all one and drawn, against dividends that
// are drawn, that differ from the divisor by a few units and that are the ends of
// the range; exponents inside and outside the range handled.  Prints the number
// of differences per operation.
#include <cstdio>

#include <cuda_runtime.h>

#include "eph_softfp.cuh"

using namespace ephgb::soft;

__device__ u64 draw(u64 &s) {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}

__device__ bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }

__global__ void check(unsigned long long *bad) {
  const u64 top = (u64)(blockIdx.x * blockDim.x + threadIdx.x);  // < 2^23
  u64 s = 88172645463325252ull ^ (top * 0x9E3779B97F4A7C15ull);
  for (int k = 0; k < 4; ++k) draw(s);
  const u64 M = 0xfffffffffffffull;
  for (int rest = 0; rest < 4; ++rest) {
    const u64 low = rest == 0 ? 0 : (rest == 1 ? 0x1fffffffull : draw(s) & 0x1fffffffull);
    const u64 mb = (top << 29) | low;
    for (int k = 0; k < 12; ++k) {
      u64 ma = draw(s) & M;
      if (k == 0) ma = 0;
      if (k == 1) ma = M;
      if (k >= 2 && k < 7) ma = (mb + (u64)(k - 4)) & M;
      u64 ea = 900 + draw(s) % 250, eb = 900 + draw(s) % 250;
      if (k == 10) ea = (draw(s) & 1) ? 511 + draw(s) % 5 : 1531 + draw(s) % 5;
      if (k == 11) eb = draw(s) % 2048, ea = draw(s) % 2048;
      const double a = from_bits((draw(s) << 63) | (ea << 52) | ma), b = from_bits((draw(s) << 63) | (eb << 52) | mb);
      if (!same(div(a, divisor(b)), a / b)) atomicAdd(bad + 1, 1ull);
      if (!same(mul(a, b), a * b)) atomicAdd(bad, 1ull);
    }
  }
}

int main() {
  unsigned long long *bad = nullptr, h[2] = {~0ull, ~0ull};
  if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMemset(bad, 0, sizeof(h)) != cudaSuccess) return 1;
  check<<<1 << 15, 256>>>(bad);
  if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  std::printf("mul %llu\ndiv %llu\n", h[0], h[1]);
  return 0;
}
