// div_rn (epic_gb300/csrc/fix_math.cuh) against the binary64 division, bit for bit: every leading
// 24-bit pattern of the divisor's significand (the reciprocal seed's whole domain) with several
// dividends each, quotients next to rounding boundaries and to powers of two, and operands at the
// ends of the range, subnormal, zero, infinite and NaN.
#include <cstdio>
#include "fix_math.cuh"
using namespace epic;

__device__ unsigned long long mix(unsigned long long x) {   // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ void check(double a, double b, unsigned long long *bad) {
  const double r = div_rn(a, b), w = a / b;
  if (__double_as_longlong(r) != __double_as_longlong(w) && !(r != r && w != w)) atomicAdd(bad, 1ull);
}
__global__ void k_div(int seed, unsigned long long *bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23: the 23 bits below the leading one
  const unsigned long long m52 = 0x000FFFFFFFFFFFFFull;
  unsigned long long g = mix(((unsigned long long)seed << 32) | i);
  auto dbl = [](unsigned long long u) { return __longlong_as_double((long long)u); };
  for (int q = 0; q < 6; q++) {
    g = mix(g);
    const unsigned long long low = q == 0 ? 0 : (q == 1 ? (1ull << 29) - 1 : g & ((1ull << 29) - 1));
    const unsigned long long sb = ((unsigned long long)i << 29) | low;
    const double b = dbl((1023ull << 52) | sb);
    g = mix(g);
    check(dbl(((1000ull + g % 46) << 52) | (mix(g) & m52)), -b, bad);            // any dividend
    check(dbl((1023ull << 52) | ((sb + (g % 5) - 2) & m52)), b, bad);            // quotient near 1
    const double c = dbl((1023ull << 52) | (mix(g + 1) & m52));
    check(dbl((unsigned long long)__double_as_longlong(b * c) + (g % 3) - 1), b, bad);   // near a double
    check(mix(g + 2) & 1 ? 0. : -0., b, bad);
    check(dbl(mix(g + 3)), dbl(mix(g + 4)), bad);                                // any bits at all
    check(dbl(mix(g + 5) & ~(0x7FFull << 52)), b, bad);                          // subnormal
    check(b, dbl(mix(g + 6) & ~(0x7FFull << 52)), bad);
    check(dbl(mix(g + 7) | (0x7FEull << 52)), b * 0.5, bad);                     // overflow, infinity, NaN
    check(dbl((1ull << 52) | (mix(g + 8) & m52)), b, bad);                       // smallest normal quotients
    check(b, dbl((0x7FEull << 52) | (mix(g + 9) & m52)), bad);
  }
  if (i < 2) check(i ? 1. : 0., 0., bad);
}
int main() {
  unsigned long long *bad = nullptr, h = 0;
  if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMemset(bad, 0, sizeof(h)) != cudaSuccess) return 2;
  for (int seed = 0; seed < 4; seed++) k_div<<<(1 << 23) / 256, 256>>>(seed, bad);
  if (cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("div_rn mismatches: %llu\n", h);
  return h != 0;
}
