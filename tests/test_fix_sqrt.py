"""The integer-pipe square root (epic_gb300/csrc/fix_math.cuh) from estimates anywhere within the bound that its
comment states: host-compiled, against the C library's root (correctly rounded)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "epic_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#define __host__
#define __device__
#define __forceinline__ inline
#include "fix_math.cuh"
using namespace epic;
static uint64_t mix(uint64_t x) {   // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
int main() {
  const double bound = std::exp2(-21.5);
  long bad = 0;
  for (uint64_t i = 0; i < 6000000; i++) {
    const uint64_t g = mix(i), h = mix(g);
    uint64_t m = g & 0x000FFFFFFFFFFFFFull;
    double x, rel = bound * (2. * (double)(h >> 11) * 0x1p-53 - 1.);
    if (i % 4 == 1) m >>= h & 31;                     // next to 1 and 2
    if (i % 4 == 2) m = 0x000FFFFFFFFFFFFFull ^ (m >> (h & 31));   // next to 2 and 4
    if (i % 8 == 3) rel = h & 1 ? bound : -bound;
    uint64_t u = (1023ull + (h >> 60 & 1)) << 52 | m;
    std::memcpy(&x, &u, 8);
    if (i % 4 == 3) {                                 // next to squares of numbers half way between two
      const long double c = 1.0L + (long double)(m >> 11) * 0x1p-41L + 0x1p-53L;
      x = (double)(c * c);
    }
    std::memcpy(&u, &x, 8);
    const uint32_t odd = ((uint32_t)(u >> 52) & 1u) ^ 1u;
    const uint64_t v = ((u & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << (10 + odd);
    const double y = 4294967296. / std::sqrt((double)(uint32_t)(v >> 32) * 0x1p-30) * (1. + rel);
    const uint32_t y0 = y < 4294967295. ? (uint32_t)y : 4294967295u;
    const double got = std::ldexp((double)sqrt_steps(v, y0), -52), want = std::sqrt(x);
    bad += got != want;
  }
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


def test_root_from_every_estimate_in_the_bound(tmp_path):
    src, exe = tmp_path / "root.cpp", str(tmp_path / "root")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
