// log2 and exp2 in 64- and 128-bit fixed point on the integer pipe: the fast paths of the
// correctly rounded log, exp and pow (dd_math.cuh).  Below them div_rn and sqrt_rn, the correctly
// rounded quotient and root on the same pipe.
//
// GB300 retires under two binary64 operations a clock and SM: a warp instruction takes 19 clocks (64 in a
// chain), a 32 x 32 -> 64 bit multiply-add one or two.  The double-double fast paths these replace
// spend about 125 binary64 operations on a pow (2000 clocks a warp); these spend about 200 integer
// ones.  Measured on a GB300 (FP64 form): 12 steps of 128x64x20 with its transfers 29.7 -> 20.5 ms, 3
// steps of 256x128x32 43.3 -> 29.1 ms; the column kernels that evaluate them (set_p2etc,
// store_pgrad_vars, calc_w) were two thirds of the step.  The results are the same bits: each path only
// returns a value whose whole error interval rounds to one binary64 number, and leaves the rest to the
// double-double evaluation.
//
// Methods (textbook fixed point): log2(x) = e + log2(c) + log2(1 + r) with a table over the ten
// leading bits of the significand m of 1/c rounded up to 20 bits, so that 1 + r = m / c is the
// product's low 64 bits, exact, with 0 <= r < 2^-10 (1 + 2^-8); log(1 + r) by its Taylor series, each
// coefficient in the width its term needs.  2^f = 2^(j/1024) (1 + g), g = 2^r - 1 by its Taylor
// series in r ln 2.  The tables are built on the host from the double-double series of dd_math.cuh.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define EPIC_COLD __noinline__
#else
#define EPIC_COLD __attribute__((noinline))
#endif

namespace epic {

struct u128 { uint64_t hi, lo; };

__host__ __device__ __forceinline__ uint64_t mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
__host__ __device__ __forceinline__ int clz64(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
__host__ __device__ __forceinline__ u128 add128(u128 a, u128 b) {
  const uint64_t lo = a.lo + b.lo;
  return {a.hi + b.hi + (lo < a.lo ? 1u : 0u), lo};
}
__host__ __device__ __forceinline__ u128 neg128(u128 a) { return {~a.hi + (a.lo == 0 ? 1u : 0u), 0ull - a.lo}; }
__host__ __device__ __forceinline__ u128 shr128(u128 a, int s) {   // 0 < s < 64
  return {a.hi >> s, (a.hi << (64 - s)) | (a.lo >> s)};
}
__host__ __device__ __forceinline__ u128 shl128(u128 a, int s) {   // 0 < s < 64
  return {(a.hi << s) | (a.lo >> (64 - s)), a.lo << s};
}
// (a * b) / 2^64, rounded down to at most two units too small
__host__ __device__ __forceinline__ u128 mul128_64(u128 a, uint64_t b) {
  return add128({mulhi64(a.hi, b), a.hi * b}, {0, mulhi64(a.lo, b)});
}

constexpr int FIX_N = 1024;
struct FixTable {
  uint32_t inv[FIX_N];   // 2^20 / (1 + i/1024), rounded up
  u128 lg[FIX_N];        // -log2(inv[i] / 2^20) in units of 2^-96
  u128 e2[FIX_N];        // 2^(j/1024) in units of 2^-127
};

constexpr uint64_t FIX_LOG2E_HI = 0xb8aa3b295c17f0bbull, FIX_LOG2E_LO = 0xbe87fed0691d3e89ull;   // 1/ln 2, units of 2^-127
constexpr uint64_t FIX_LN2_HI = 0xb17217f7d1cf79abull, FIX_LN2_LO = 0xc9e3b39803f2f6afull;       // ln 2, units of 2^-128

// log2(x) in units of 2^-96, two's complement, for a positive normal x of bits u.  |error| < 2^-79:
// r is exact; r/ln 2 is kept to 2^-130; q = r - log(1 + r) = r^2 (1/2 - r/3 + ... + r^5/7) to 2^-81 (the
// r^8 term dropped is below 2^-83); the table to 2^-97.
__host__ __device__ __forceinline__ u128 fix_log2(uint64_t u, const FixTable &T) {
  const int i = (int)(u >> 42) & (FIX_N - 1);
  const uint64_t m = (u & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  const uint64_t r72 = m * T.inv[i];           // r in units of 2^-72 (the 1 of 1 + r is 2^72: gone)
  const u128 lc = T.lg[i];
  const uint64_t r = r72 << 1;                 // units of 2^-73, below 2^63.02
  const uint32_t r32 = (uint32_t)(r >> 32);    // units of 2^-41
  const uint32_t t4 = 0xaaaaaaabu - (mulhi32(r32, 0x92492492u) >> 9);            // 1/6 - r/7, 2^-34
  const uint32_t t3 = 0xcccccccdu - (mulhi32(r32, t4) >> 9);                     // 1/5 - r t4, 2^-34
  const uint64_t t2 = 0x8000000000000000ull - (((uint64_t)r32 * t3) >> 10);      // 1/4 - r t3, 2^-65
  const uint64_t t1 = 0xaaaaaaaaaaaaaaabull - (mulhi64(r, t2) >> 9);             // 1/3 - r t2, 2^-65
  const uint64_t w = 0x8000000000000000ull - (mulhi64(r, t1) >> 10);             // 1/2 - r t1, 2^-64
  const uint64_t q = mulhi64(mulhi64(r, r), w);                                  // 2^-82
  const uint64_t cq = mulhi64(q, FIX_LOG2E_HI);                                  // q / ln 2, 2^-81
  // r / ln 2 in units of 2^-135, then of 2^-96
  const u128 cr = shr128(add128({mulhi64(r72, FIX_LOG2E_HI), r72 * FIX_LOG2E_HI}, {0, mulhi64(r72, FIX_LOG2E_LO)}), 39);
  u128 v = add128(lc, cr);
  const uint64_t sub_lo = cq << 15;
  v.hi -= (cq >> 49) + (v.lo < sub_lo ? 1u : 0u);
  v.lo -= sub_lo;
  v.hi += (uint64_t)(int64_t)((int)(u >> 52) - 1023) << 32;
  return v;
}

// Round sig / 2^127 (sig.hi's top bit set: a number in [1, 2)) times 2^n to binary64, if every number
// within err units of 2^-116 of it rounds the same way; n in the normal range.
__host__ __device__ __forceinline__ bool fix_round(u128 sig, int n, uint64_t err, uint64_t &bits) {
  const uint64_t rem = (sig.hi << 53) | (sig.lo >> 11);   // below the last place, in 2^-64 of it
  bits = ((uint64_t)(n + 1022) << 52) + (sig.hi >> 11) + (rem >> 63);
  return rem - 0x8000000000000000ull + err > 2 * err && (int64_t)sig.hi < 0;
}

// 2^z for z in units of 2^-96, two's complement, |z| < 1000: rounded to binary64, or false where the
// rounding is not certain.  rel: what z's own error adds, in units of 2^-116 of the result.  The
// evaluation's relative error is below 2^-70: g's terms round down by less than 2^-72 in all, its
// product with the table entry by 2^-73, and the table entry's part below 2^-63 adds 2^-73.5.
__host__ __device__ __forceinline__ bool fix_exp2(u128 z, uint64_t rel, const FixTable &T, uint64_t &bits) {
  const int n = (int)((int64_t)z.hi >> 32);
  const uint32_t f = (uint32_t)z.hi;
  const uint64_t r = ((uint64_t)(f & 0x3fffffu) << 42) | (z.lo >> 22);           // 2^-74
  const u128 t = T.e2[f >> 22];
  const uint64_t a = mulhi64(r, FIX_LN2_HI);                                     // r ln 2, 2^-74
  const uint32_t a32 = (uint32_t)(a >> 32);                                      // 2^-42
  const uint32_t s1 = 0x88888889u + (mulhi32(a32, 0xb60b60b6u) >> 13);           // 1/120 + a/720, 2^-38
  const uint32_t s2 = 0xaaaaaaabu + (mulhi32(a32, s1) >> 12);                    // 1/24 + a s1, 2^-36
  const uint64_t s3 = 0xaaaaaaaaaaaaaaabull + (((uint64_t)a32 * s2) >> 12);      // 1/6 + a s2, 2^-66
  const uint64_t a2 = mulhi64(a, a);                                             // 2^-84
  const uint64_t a3s = mulhi64(mulhi64(a2, a), s3);                              // a^3 s3, 2^-96
  const uint64_t g = a + (((a2 >> 1) + (a3s >> 12)) >> 10);                      // 2^r - 1, 2^-74
  const uint64_t p = mulhi64(t.hi, g);                                           // 2^-73
  return fix_round(add128(t, {p >> 10, p << 54}), n, (1ull << 47) + rel, bits);
}

// ---- division ----

// A reciprocal estimate 2^31 y of b in [1, 2), y within 2^-22 of 1/b.
__host__ __device__ __forceinline__ uint32_t recip31(uint32_t b24) {   // b's leading 24 bits
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f000000u + b24)));
  const uint32_t q = __float2uint_rz(y * 2147483648.f);
#else
  const uint32_t q = (uint32_t)(0x1p54 / (double)b24);
#endif
  return q < 0x7fffffffu ? q : 0x7fffffffu;
}

static __host__ __device__ EPIC_COLD double div_cold(double a, double b) { return a / b; }

// a / b rounded to nearest, the IEEE quotient, by long division of the significands in two digits of
// 26 bits with a 32-bit reciprocal: about 60 integer instructions (30 clocks a warp) where the
// binary64 pipe takes about ten operations (160 clocks).  Measured (FP64 form): 12 steps of 128x64x20
// with transfers 20.5 -> 17.2 ms, 3 steps of 256x128x32 29.1 -> 23.5 ms.  The second digit is within 0.71 of the exact
// quotient, so one comparison of the exact remainder with half the divisor rounds it; a quotient of
// two 53-bit significands is never half way.  Zero dividends are answered here too (differences of
// equal values are common in the fields); infinities, NaN, subnormals, zero divisors and quotients at
// the ends of the range go to the division itself.
__host__ __device__ __forceinline__ double div_rn(double a, double b) {
  uint64_t ua, ub;
#ifdef __CUDA_ARCH__
  ua = (uint64_t)__double_as_longlong(a);
  ub = (uint64_t)__double_as_longlong(b);
#else
  memcpy(&ua, &a, 8);
  memcpy(&ub, &b, 8);
#endif
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7FFu, eb = (uint32_t)(ub >> 52) & 0x7FFu;
  const uint64_t ma = (ua & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  const uint64_t mb = (ub & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  const int s = ma < mb ? 1 : 0;               // the significands' quotient 2^s ma / mb in [1, 2)
  const uint32_t e = ea - eb + 1023u - (uint32_t)s;
  const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
  const bool zero = (ua << 1) == 0 && eb - 1u < 2046u;
  if (!zero && (ea - 1u >= 2046u || eb - 1u >= 2046u || e - 1u >= 2045u)) return div_cold(a, b);
  const uint32_t y0 = recip31((uint32_t)(mb >> 29));                          // 1/b, units of 2^-31
  const int t = (int)(((int64_t)1 << 52) - (int64_t)(((mb >> 21) * (uint64_t)y0) >> 10));   // 1 - b y0, 2^-52
  const uint32_t y = 2u * y0 + (uint32_t)(((int64_t)t * (int)y0) >> 51);      // one Newton step, 2^-32
  const uint32_t q1 = mulhi32((uint32_t)(ma >> (22 - s)), y) >> 4;            // the quotient, 2^-26
  const int64_t r1 = (int64_t)((ma << (26 + s)) - mb * q1);
  const int q2 = (int)(((int64_t)(int)(r1 >> 23) * (int64_t)(uint64_t)y + ((int64_t)1 << 34)) >> 35);   // 2^-52
  const int64_t r2 = 2 * (int64_t)(((uint64_t)r1 << 26) - mb * (uint64_t)(int64_t)q2);
  uint64_t q = ((uint64_t)q1 << 26) + (uint64_t)(int64_t)q2;
  q += r2 > (int64_t)mb ? 1 : 0;
  q -= r2 < -(int64_t)mb ? 1 : 0;
  const uint64_t u = (zero ? 0 : ((uint64_t)(e - 1u) << 52) + q) | sign;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double r;
  memcpy(&r, &u, 8);
  return r;
#endif
}

// ---- square root ----

// A reciprocal square root estimate 2^32 y of v in [1, 4), y within 2^-21.5 of 1/sqrt(v), relative: the
// instruction's documented 2^-22.9, v's rounding to binary32 (2^-25), the product's (2^-24) and the factor
// 1 - 2^-24 together are below 2^-21.7.  An estimate above the largest 32-bit number becomes that number (the
// conversion saturates), which is nearer.
__host__ __device__ __forceinline__ uint32_t rsqrt32(uint32_t v30) {   // v in units of 2^-30
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint2float_rn(v30) * 9.31322574615478515625e-10f));
  return __float2uint_rz(y * 4294967040.f);
#else
  return (uint32_t)(4294967040. / __builtin_sqrt((double)v30 * 0x1p-30));
#endif
}

static __host__ __device__ EPIC_COLD double sqrt_cold(double x) {
#ifdef __CUDA_ARCH__
  return ::sqrt(x);
#else
  return __builtin_sqrt(x);
#endif
}

// sqrt(v) of v in [1, 4), in units of 2^-62, rounded to nearest in units of 2^-52, from an estimate y0 of
// 2^32 / sqrt(v) within 2^-21.5.  One Newton step leaves y within 2^-30 (its own error 2^-42, the dropped bits
// of v and of v y0 add up to 2^-30 y, the last shift takes 2^-32); s = v y is then within 2^-28 of the
// root, so v - s^2 is at most 2^-26 and its top 32 bits fit an int; and s + (v - s^2) y / 2 with the exact
// v - s^2 is off by less than 2^-57 (second order) + 2^-55 (y's error) + 2^-57 (the int's dropped bits), and
// the sum's rounding adds half a unit: within 0.75 units, so the exact remainder of the result moves it by at most
// one; a root is never half way.  tests/test_fix_sqrt.py moves the estimate to the ends of its bound.
__host__ __device__ __forceinline__ uint64_t sqrt_steps(uint64_t v, uint32_t y0) {
  const uint32_t vh = (uint32_t)(v >> 32);                                                  // 2^-30
  const uint32_t vy = mulhi32(vh, y0);                                                      // v y0, 2^-30
  const int t = (int)(((int64_t)1 << 46) - (int64_t)(((uint64_t)vy * y0) >> 16));           // 1 - v y0^2, 2^-46
  const uint32_t yd = y0 + (uint32_t)(int32_t)(((int64_t)t * (int64_t)(uint64_t)y0) >> 47);
  const uint32_t y = yd < y0 && t > 0 ? 0xffffffffu : yd;                                   // v = 1: y stays below 1
  const uint32_t s = mulhi32(vh, y);                                                        // 2^-30
  const int64_t r = (int64_t)(v - ((uint64_t)s * s << 2));                                  // v - s^2, 2^-62, exact
  const int64_t d = ((int64_t)(int)(r >> 6) * (int64_t)(uint64_t)y + ((int64_t)1 << 36)) >> 37;   // r y / 2, 2^-52
  uint64_t q = ((uint64_t)s << 22) + (uint64_t)d;
  const int64_t rem = (int64_t)((v << 42) - q * q);                                         // 2^-104, small
  q += rem > (int64_t)q ? 1 : 0;
  q -= rem <= -(int64_t)q ? 1 : 0;
  return q;
}

// sqrt(x) rounded to nearest on the integer pipe: about 45 integer instructions where the binary64
// pipe takes about ten operations, 16 clocks each.  v in [1, 4) is x over an even power of 2.  Zeros are
// answered here (one side of a split velocity always is); subnormals, negative numbers, infinities and NaN go
// to the function itself.
__host__ __device__ __forceinline__ double sqrt_rn(double x) {
  uint64_t u;
#ifdef __CUDA_ARCH__
  u = (uint64_t)__double_as_longlong(x);
#else
  memcpy(&u, &x, 8);
#endif
  const uint32_t e = (uint32_t)(u >> 52);   // with the sign: above 2047 for a negative number
  const bool zero = (u << 1) == 0;
  if (!zero && e - 1u >= 2046u) return sqrt_cold(x);
  const uint32_t odd = (e & 1u) ^ 1u;       // an even biased exponent is an odd power of 2
  const uint64_t v = ((u & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << (10 + odd);   // 2^-62
  const uint64_t q = sqrt_steps(v, rsqrt32((uint32_t)(v >> 32)));
  const uint64_t w = zero ? u : ((uint64_t)((e + 1021u) >> 1) << 52) + q;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)w);
#else
  double res;
  memcpy(&res, &w, 8);
  return res;
#endif
}

}  // namespace epic
