// sqrt_rn (epic_gb300/csrc/fix_math.cuh) against the binary64 square root, bit for bit: every leading
// 23-bit pattern of the argument over both exponent parities (the seed's whole domain), arguments next
// to squares, to powers of two and to squares of half-way points, and operands at the ends of the range,
// subnormal, zero, negative, infinite and NaN.
#include <cstdio>
#include "fix_math.cuh"
using namespace epic;

__device__ unsigned long long mix(unsigned long long x) {   // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ void check(double a, unsigned long long *bad) {
  const double r = sqrt_rn(a), w = sqrt(a);
  if (__double_as_longlong(r) != __double_as_longlong(w) && !(r != r && w != w)) atomicAdd(bad, 1ull);
}
__global__ void k_sqrt(int seed, unsigned long long *bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23
  const unsigned long long m52 = 0x000FFFFFFFFFFFFFull;
  unsigned long long g = mix(((unsigned long long)seed << 32) | i);
  auto dbl = [](unsigned long long u) { return __longlong_as_double((long long)u); };
  for (int q = 0; q < 6; q++) {
    g = mix(g);
    const unsigned long long low = q == 0 ? 0 : (q == 1 ? (1ull << 29) - 1 : g & ((1ull << 29) - 1));
    const unsigned long long sb = ((unsigned long long)i << 29) | low;
    const double b = dbl((1023ull << 52) | sb);
    check(b, bad);
    check(2. * b, bad);
    check(dbl(((1ull + mix(g) % 2046) << 52) | sb), bad);                                         // any exponent
    check(dbl((unsigned long long)__double_as_longlong(b * b) + (g % 5) - 2), bad);               // near a square
    check(dbl((((1022ull + (g & 3)) << 52) | (g >> 60)) - ((g >> 56) & 15)), bad);                // near a power of 2
    const double c = dbl((1023ull << 52) | (sb & ~((1ull << 26) - 1)));                           // exact squares
    check(c * c, bad);
    check(mix(g + 2) & 1 ? 0. : -0., bad);
    check(dbl(mix(g + 3)), bad);                                                                  // any bits at all
    check(dbl(mix(g + 4) & m52), bad);                                                            // subnormal
    check(dbl((0x7FEull << 52) | (mix(g + 5) & ((1ull << 53) - 1))), bad);                        // largest, infinity, NaN
  }
}
int main() {
  unsigned long long *bad = nullptr, h = 0;
  if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMemset(bad, 0, sizeof(h)) != cudaSuccess) return 2;
  for (int seed = 0; seed < 4; seed++) k_sqrt<<<(1 << 23) / 256, 256>>>(seed, bad);
  if (cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("sqrt_rn mismatches: %llu\n", h);
  return h != 0;
}
