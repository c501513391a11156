// fastmath.cuh — FP64 exp, exp10, log, reciprocal, division, reciprocal
// square root and arc tangent that spend few or no FP64 instructions.
//
// GB300 issues FP64 at 1/64 of its FP32 rate (a measured 1.0 TFLOP/s FMA): a
// warp's FP64 instruction holds the SM's pipe for 16 cycles, in which the four
// schedulers could issue 64 others, and an FP64 compare, min/max or conversion
// costs as much as an FMA.  The microphysics kernels need a few dozen of these
// functions per grid point and ran the FP64 pipe at 78-85 % with 80-88 % of
// the issue slots idle, so the functions work in 64-bit fixed point on the
// integer pipe (32 x 32 -> 64-bit multiplies), to a few units of 2^-60 of the
// result, rounded once: a function of ~70 integer instructions in place of 6-9
// FP64 ones is about 1/6 of their cost, and more accurate (0.53 ulp instead of
// about 1).  256x256x90, exp / log on FP64 -> integer: rain_ice 12.01 -> 9.60
// ms, adjoint 24.8 -> 19.1 ms; ice_adjust (4.1 M points) 2.12 -> 1.61 ms;
// sedimentation (65,535 x 87) 4.27 -> 2.88 ms.
//
//   fexp   after P. T. P. Tang, "Table-driven implementation of the
//          exponential function in IEEE floating-point arithmetic", ACM TOMS
//          15(2), 1989: x = k ln2/512 + r, 0 < r < 2^-8.8 (k from an FP32
//          estimate, one low so that every term of the series is positive;
//          r exact modulo 2^-6 in units of 2^-70); e^x = 2^(k/512) e^r,
//          2^(j/512) tabulated to 62 bits, e^r - 1 by its Taylor series to
//          r^5.  Within 0.52 ulp.
//   fexp10 the same with log10(2)/512 and r scaled by ln 10.
//   flog   after P. T. P. Tang, "Table-driven implementation of the logarithm
//          function in IEEE floating-point arithmetic", ACM TOMS 16(4), 1990:
//          x = 2^e z, z in [1, 2) in 512 intervals; per interval an integer
//          c = ceil(2048 / lower end) makes r = z c/2048 - 1 exact, 0 <= r <
//          2^-8.4; log x = e ln2 - log(c/2048) + log1p(r), log1p by its Taylor
//          series to r^7, the sum in 96 bits (2^-72).  Within 0.54 ulp.  Within
//          2^-8 of x = 1, where the sum cancels, log1p(x - 1) in FP64.
//   frcp   1/d and fdiv a/b, the IEEE results bit for bit, in integer
//          arithmetic (no FP64 operation): with d = x 2^k, x in [1, 2), the
//          hardware's FP32 reciprocal y0 of x (24 bits, |eps| = |1 - x y0| <
//          2^-21), one Newton-Raphson step with its quadratic term, y0 (1 +
//          eps + eps^2), in 64-bit fixed point (eps exact, remainder eps^3 <
//          2^-63), the significand (of a times it) rounded to 53 bits, and
//          the rounding settled by the exact remainder (a - q b modulo 2^64).
//          A quotient of doubles is never halfway between two doubles, so the
//          sign of |r| - |b|/2 decides; the seed's error cannot reach the
//          result.  In place of 3 / 7 FP64 operations of a reciprocal /
//          rounded division: rain_ice 13.60 -> 12.01 ms, adjoint 26.3 ->
//          24.8 ms (256x256x90).  Where an operand is zero, subnormal, infinite or NaN, or
//          the result leaves the normal range, the IEEE division.
//   frsqrt 1/sqrt(d) in the same way: d = x 4^k, x in [1, 4); y0 = the FP32
//          reciprocal of the FP32 square root of x (24 bits, |eps| = |1 - x
//          y0^2| < 2^-21, exact in integers), y0 (1 + eps/2 + 3 eps^2/8), the
//          series of (1 - eps)^(-1/2) to its quadratic term (remainder below
//          2^-64), rounded once: within 0.51 ulp, no FP64 operation.
//          fsqrt_rn: sqrt(d), the IEEE result bit for bit, from it.
//   fatan  reduction to y in (0, 1] by atan(x) = pi/2 - atan(1/x), then
//          atan(y) = atan(c) + atan(r), c = j/64 the nearest table point,
//          r = (y - c)/(1 + y c) (|r| <= 1/128), atan(r) by its Taylor series
//          to r^7; atan(c) and pi/2 - atan(c) tabulated; in 64-bit fixed
//          point, units of 2^-64 where the result is below 1 (table and shift
//          each rounded to 2^-65, r within 2^-66: below 0.04 ulp of the
//          smallest result, 2^-7) and 2^-62 above; rounded once, no FP64
//          operation.  Below 2^-7 the series in FP64.
//
// Accuracy: within 2 ulp (tests compare the host build of this code with
// 200-bit mpmath values).  Every FP64 and FP32 operation is an explicit fma or
// a separately rounded add/multiply, and the tests find the device build equal
// to the host build bit for bit, but for the last bit of fatan: its quotient is
// not settled, and the device's seed of it is the hardware's approximation (the
// host's the rounded reciprocal).  Special inputs (NaN, infinities, zero,
// negative, subnormal, overflow and underflow ranges) leave the fast path
// through one integer test and get the IEEE results of exp/log.
#pragma once

#include <stdint.h>
#include <string.h>
#if !defined(__CUDACC__)
#include <cmath>
#endif

#include "fastmath_tables.h"

#if defined(__CUDACC__)
#define FM_HD __host__ __device__ __forceinline__
// exp, exp10, log, the reciprocal and the rounded division are called from
// dozens of sites of the large point kernels: one out-of-line copy per
// kernel keeps those kernels' code in the instruction cache (rain_ice 172.5
// -> 171.5 ms and sedimentation 46.1 -> 44.7 ms per launch at 1024x1024x90
// for exp / log; rain_ice 162.4 -> 159.2 ms for the reciprocal, 160.7 ms
// for the division)
#define FM_NI static __host__ __device__ __noinline__
#else
#define FM_HD inline
#define FM_NI static inline
#endif

namespace fm {

struct alignas(16) AtanEntry { uint64_t at, co; };   // atan(j/64), 2^-64; pi/2 - atan(j/64), 2^-62
struct alignas(16) LogEntry { uint32_t c, n0, n1, n2; };

#if defined(__CUDA_ARCH__)
__device__ const uint64_t kExpTable[512] = FM_EXP_TABLE_INIT;
__device__ const LogEntry kLogTable[512] = FM_LOG_TABLE_INIT;
__device__ const AtanEntry kAtanTable[65] = FM_ATAN_TABLE_INIT;
__device__ __forceinline__ AtanEntry atan_entry(uint32_t j)
{
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(kAtanTable) + j);
  return {v.x, v.y};
}
__device__ __forceinline__ float rcpf_(float x) { return __frcp_rn(x); }
__device__ __forceinline__ float sqrtf_(float x) { return __fsqrt_rn(x); }
__device__ __forceinline__ uint64_t exp_entry(uint32_t j)
{
  return __ldg(reinterpret_cast<const unsigned long long *>(kExpTable) + j);
}
__device__ __forceinline__ LogEntry log_entry(uint32_t i)
{
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(kLogTable) + i);
  return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ uint32_t funnel_l_(uint32_t lo, uint32_t hi, uint32_t n) { return __funnelshift_lc(lo, hi, n); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fmaf_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mulf_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ int64_t bits_(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double from_bits_(int64_t b) { return __longlong_as_double(b); }
__device__ __forceinline__ int32_t fbits_(float x) { return __float_as_int(x); }
__device__ __forceinline__ float ffrom_bits_(int32_t b) { return __int_as_float(b); }
__device__ __forceinline__ int clz32_(uint32_t v) { return __clz((int)v); }
__device__ __forceinline__ uint32_t hi_(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t lo_(double x) { return (uint32_t)__double2loint(x); }
__device__ __forceinline__ uint32_t mulhi_(uint32_t a, uint32_t b) { return __umulhi(a, b); }
// 1/x within 2^-22 for the integer reciprocal (its error cannot reach a result)
__device__ __forceinline__ float rcp_seed_(float x)
{
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
#else
static const uint64_t kExpTable[512] = FM_EXP_TABLE_INIT;
static const LogEntry kLogTable[512] = FM_LOG_TABLE_INIT;
static const AtanEntry kAtanTable[65] = FM_ATAN_TABLE_INIT;
inline AtanEntry atan_entry(uint32_t j) { return kAtanTable[j]; }
inline float rcpf_(float x) { volatile float r = 1.0f / x; return r; }
inline float sqrtf_(float x) { volatile float r = std::sqrt(x); return r; }
inline uint64_t exp_entry(uint32_t j) { return kExpTable[j]; }
inline LogEntry log_entry(uint32_t i) { return kLogTable[i]; }
inline uint32_t funnel_l_(uint32_t lo, uint32_t hi, uint32_t n)
{
  return n >= 32 ? lo : (uint32_t)((((uint64_t)hi << 32 | lo) << n) >> 32);
}
inline double fma_(double a, double b, double c) { return std::fma(a, b, c); }
inline double add_(double a, double b) { volatile double s = a + b; return s; }
inline double mul_(double a, double b) { volatile double s = a * b; return s; }
inline float fmaf_(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float mulf_(float a, float b) { volatile float s = a * b; return s; }
inline int64_t bits_(double x) { int64_t b; memcpy(&b, &x, 8); return b; }
inline double from_bits_(int64_t b) { double x; memcpy(&x, &b, 8); return x; }
inline int32_t fbits_(float x) { int32_t b; memcpy(&b, &x, 4); return b; }
inline float ffrom_bits_(int32_t b) { float x; memcpy(&x, &b, 4); return x; }
inline int clz32_(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline uint32_t hi_(double x) { return (uint32_t)((uint64_t)bits_(x) >> 32); }
inline uint32_t lo_(double x) { return (uint32_t)bits_(x); }
inline uint32_t mulhi_(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// (FM_HOST_SEED_ULPS: the tests move the seed by what the device's may be off)
#ifndef FM_HOST_SEED_ULPS
#define FM_HOST_SEED_ULPS 0
#endif
inline float rcp_seed_(float x) { return ffrom_bits_(fbits_(rcpf_(x)) + FM_HOST_SEED_ULPS); }
#endif

// double -> float by truncation of the significand, with integer operations
// only; magnitudes below 2^-126 become zero.  For the small high-order terms
// computed in FP32 the 2^-23 relative error is far below what they need.
FM_HD float to_f32(double x)
{
  const int64_t b = bits_(x);
  const int32_t e = (int32_t)((b >> 52) & 0x7ff) - 896;        // float biased exponent
  const int32_t s = (int32_t)((uint64_t)b >> 32) & (int32_t)0x80000000;
  if (e <= 0) return ffrom_bits_(s);
  return ffrom_bits_(s | (e << 23) | (int32_t)((b >> 29) & 0x7fffff));
}

// float -> double, exact, with integer operations only (float zero and
// subnormals give zero).
FM_HD double to_f64(float x)
{
  const int32_t b = fbits_(x);
  const int32_t e = (b >> 23) & 0xff;
  const int64_t s = (int64_t)((uint64_t)((uint32_t)b & 0x80000000u) << 32);
  if (e == 0) return from_bits_(s);
  return from_bits_(s | ((int64_t)(e + 896) << 52) | ((int64_t)(b & 0x7fffff) << 29));
}

// int -> double, exact (|k| < 2^31), with integer operations only.
FM_HD double i2d(int32_t k)
{
  if (k == 0) return 0.0;
  const int64_t s = k < 0 ? (int64_t)(1ULL << 63) : 0;
  const uint32_t a = k < 0 ? (uint32_t)(-(int64_t)k) : (uint32_t)k;
  const int n = 31 - clz32_(a);                                  // index of the leading bit
  const int64_t mant = ((int64_t)a << (52 - n)) & 0x000fffffffffffffLL;
  return from_bits_(s | ((int64_t)(1023 + n) << 52) | mant);
}

// hi : lo of a 64 x 64-bit product's upper half, without the carry of the
// lowest partial product (at most two units low).
FM_HD uint64_t mulhi64_(uint64_t a, uint64_t b)
{
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + mulhi_(ah, bl) + mulhi_(al, bh);
}

// The square of R 2^-70 in units of 2^-76 (at most two units low).
FM_HD uint64_t sqr70_(uint64_t R)
{
  const uint32_t h = (uint32_t)(R >> 32), l = (uint32_t)R;
  return (uint64_t)h * h + (((uint64_t)h * l) >> 31);
}

// x 2^70 modulo 2^64 plus `bias`, minus kb (cl + ch 2^32) 2^-32: the exact
// argument reduction of fexp / fexp10 (|x| < 1024, kb < 2^21).
FM_HD uint64_t exp_reduce_(uint32_t h, uint32_t l, uint64_t bias, uint32_t kb, uint64_t c, uint32_t clo)
{
  const uint32_t e = (h >> 20) & 0x7ffu;
  const uint64_t m = ((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | l;
  // 2^(e - 1075) m = m 2^(e - 1005) 2^-70; below 2^-18 the bits under 2^-70 drop
  const uint32_t down = 1005u - e;
  uint64_t X = e >= 1005u ? m << (e - 1005u) : (down < 64u ? m >> down : 0u);
  if ((int32_t)h < 0) X = 0u - X;
  const uint64_t kc = (uint64_t)kb * (uint32_t)c + ((uint64_t)(kb * (uint32_t)(c >> 32)) << 32);
  return X + bias - kc - mulhi_(kb, clo);
}

// 2^(k/512) e^r for r = R 2^-70 in (0, 2^-8.8), k = kb - 2^20: T + T (e^r - 1)
// with T = 2^(j/512) 2^62 from the table and
// e^r - 1 = r + r^2/2 + r^3 (1/6 + r/24 + r^2/120), all terms positive, each
// held to 2^-60 or better of the result; rounded once to 53 bits: q 2^(m - 52).
FM_HD void exp_core_(uint64_t R, uint32_t kb, uint64_t &q, int32_t &m)
{
  const uint64_t r2 = sqr70_(R);
  const uint32_t r40 = (uint32_t)(R >> 30);                       // r 2^40
  const uint32_t u = 357913941u + mulhi_(r40, 279620u);          // (1/24 + r/120) 2^33
  const uint32_t t = 2863311531u + (mulhi_(r40, u) >> 7);        // (1/6 + r/24 + ...) 2^34
  const uint32_t s = (uint32_t)(((uint64_t)r40 * t) >> 31);      // r times it, 2^43
  const uint64_t p = (R >> 6) + (r2 >> 13) + (((uint64_t)(uint32_t)(r2 >> 27) * s) >> 28);   // (e^r - 1) 2^64
  const uint64_t T = exp_entry(kb & 511u);
  const uint64_t y = T + mulhi64_(T, p);                          // [2^62, 2^63.004)
  const uint32_t ov = (uint32_t)(y >> 63);
  m = (int32_t)(kb >> 9) - 2048 + (int32_t)ov;
  q = (y + (512u << ov)) >> (10u + ov);                           // 53 bits
}

// q 2^(m - 52), rounded once more only where it is subnormal.
FM_HD double exp_scale_(uint64_t q, int32_t m)
{
  if (m >= -1022 && m <= 1022) return from_bits_((int64_t)(q + ((uint64_t)(uint32_t)(m + 1022) << 52)));
  // gradual underflow / overflow edges: scale in two steps
  const double d = from_bits_((int64_t)(q + ((uint64_t)(uint32_t)(m / 2 + 1022) << 52)));
  return mul_(d, from_bits_((int64_t)(1023 + m - m / 2) << 52));
}

// k + 2^20 with k the integer nearest x s less one (|x s| < 2^20, x as a
// float to 2^-23: k is at most 1.6 below x s, and below it).
FM_HD uint32_t exp_index_(float x, float s)
{
  const float sh = 12582912.0f;                                   // 1.5 * 2^23
  return (uint32_t)(fbits_(fmaf_(x, s, sh)) - fbits_(sh)) + 1048575u;
}

FM_HD void exp_parts_(double x, uint64_t &q, int32_t &m)
{
  const uint32_t kb = exp_index_(to_f32(x), FM_INV_L512_F);
  exp_core_(exp_reduce_(hi_(x), lo_(x), FM_L512_BIAS, kb, FM_L512_HI, FM_L512_LO), kb, q, m);
}

// e^x.
FM_NI double fexp(double x)
{
  const uint32_t h = hi_(x);
  if ((h & 0x7fffffffu) >= 0x40862e43u) {                         // |x| > 709.78, inf, NaN
    if (x != x) return x;
    if (x > 709.782712893384) return from_bits_(0x7ff0000000000000LL);
    if (x < -745.1332191019412) return 0.0;
  }
  uint64_t q;
  int32_t m;
  exp_parts_(x, q, m);
  return exp_scale_(q, m);
}

// 10^x.
FM_NI double fexp10(double x)
{
  const uint32_t h = hi_(x);
  if ((h & 0x7fffffffu) >= 0x40734413u) {                         // |x| > 308.25, inf, NaN
    if (x != x) return x;
    if (x > 308.2547155599167) return from_bits_(0x7ff0000000000000LL);
    if (x < -323.60766413161369) return 0.0;
  }
  const uint32_t kb = exp_index_(to_f32(x), FM_INV_LG512_F);
  const uint64_t r10 = exp_reduce_(h, lo_(x), FM_LG512_BIAS, kb, FM_LG512_HI, FM_LG512_LO);
  uint64_t q;
  int32_t m;
  exp_core_(mulhi64_(r10, FM_LN10_62) << 2, kb, q, m);
  return exp_scale_(q, m);
}

// log1p(r) for |r| <= 2^-8 (exact r = x - 1): r + r^2 q, q to r in FP64 and
// from r^3 on in FP32.
FM_NI double log_near1_(double x)
{
  const double r = add_(x, -1.0);
  const float rf = to_f32(r);
  float s = fmaf_(rf, -1.0f / 8.0f, 1.0f / 7.0f);
  s = fmaf_(rf, s, -1.0f / 6.0f);
  s = fmaf_(rf, s, 1.0f / 5.0f);
  double q = fma_(r, to_f64(s), -0.25);
  q = fma_(r, q, 1.0 / 3.0);
  q = fma_(r, q, -0.5);
  return fma_(mul_(r, r), q, r);
}

// log of a positive x = h : l outside log_near1_'s range, ebias = 1100 - 1023
// (less 54 for a subnormal scaled by 2^54).
FM_HD double log_core_(uint32_t h, uint32_t l, uint32_t ebias)
{
  const LogEntry t = log_entry((h >> 11) & 511u);
  const uint32_t eb = (h >> 20) + ebias;                          // e + 1100
  // r 2^70 = (z c / 2048 - 1) 2^70, exact
  const uint64_t zl = (uint64_t)l * t.c;
  const uint32_t zh = ((h & 0xfffffu) | 0x100000u) * t.c + (uint32_t)(zl >> 32) - 0x80000000u;
  const uint64_t R = (((uint64_t)zh << 32) | (uint32_t)zl) << 7;
  // log1p(r) = r - r G, G = r/2 - r^2 K, K = 1/3 - r (1/4 - r (1/5 - r (1/6 - r/7)))
  const uint64_t r2 = sqr70_(R);
  const uint32_t r40 = (uint32_t)(R >> 30);                       // r 2^40
  const uint32_t w = 715827883u - mulhi_(r40, 2396745u);         // (1/6 - r/7) 2^32
  const uint32_t u = 1717986918u - (mulhi_(r40, w) >> 7);        // 2^33
  const uint32_t v = 2147483648u - (mulhi_(r40, u) >> 8);        // 2^33
  const uint64_t K = 0x5555555555555555ull - (((uint64_t)r40 * v) >> 9);   // 2^64
  const uint64_t G = (R >> 1) - (mulhi64_(r2, K) >> 6);           // 2^70
  const uint64_t L = (R << 2) - (mulhi64_(R, G) >> 4);            // log1p(r) 2^72
  // V = eb ln2 + (table) + L in 96 bits, 2^-72
  const uint64_t s0 = (uint64_t)eb * FM_LN2_W0 + t.n0 + (uint32_t)L;
  const uint64_t s1 = (uint64_t)eb * FM_LN2_W1 + t.n1 + (uint32_t)(L >> 32) + (uint32_t)(s0 >> 32);
  const uint32_t s2 = eb * FM_LN2_W2 + t.n2 + (uint32_t)(s1 >> 32);
  // |V| (2^-72 low where negative), its 64 leading bits, rounded to 53
  const uint32_t sg = (uint32_t)((int32_t)s2 >> 31);
  const uint32_t v2 = s2 ^ sg, v1 = (uint32_t)s1 ^ sg, v0 = (uint32_t)s0 ^ sg;
  const uint32_t lz = (uint32_t)clz32_(v2);                       // 0..32: |V| >= 2^-9
  const uint64_t top = ((uint64_t)funnel_l_(v1, v2, lz) << 32) | funnel_l_(v0, v1, lz);
  const uint64_t q = (top >> 11) + ((uint32_t)(top >> 10) & 1u);
  return from_bits_((int64_t)(q + ((uint64_t)(1045u - lz) << 52) + ((uint64_t)(sg & 0x80000000u) << 32)));
}

// Natural logarithm.
FM_NI double flog(double x)
{
  uint32_t h = hi_(x), l = lo_(x);
  uint32_t ebias = 77u;                                           // 1100 - 1023
  if (h - 0x3fefe000u < 0x3000u) return log_near1_(x);            // 1 - 2^-8 <= x < 1 + 2^-8
  if (h - 0x00100000u >= 0x7fe00000u) {                           // <= 0, subnormal, inf, NaN
    if (x != x) return x;
    if (x < 0.0) return from_bits_(0x7ff8000000000000LL);
    if (x == 0.0) return from_bits_((int64_t)0xfff0000000000000ULL);
    if (h >= 0x7ff00000u) return x;                               // +inf
    x = mul_(x, 18014398509481984.0);                             // subnormal: * 2^54
    h = hi_(x);
    l = lo_(x);
    ebias = 77u - 54u;
  }
  return log_core_(h, l, ebias);
}

// Two logarithms / exponentials at once: the two dependent chains of integer
// operations overlap, where a single one leaves a warp waiting for its own
// results (used where a warp needs pairs and its latency counts).
struct Pair { double a, b; };
FM_HD bool log_plain_(double x)                                   // normal, positive, not next to 1
{
  const uint32_t h = hi_(x);
  return h - 0x00100000u < 0x7fe00000u && h - 0x3fefe000u >= 0x3000u;
}
FM_NI Pair flog2(double a, double b)
{
  if (log_plain_(a) && log_plain_(b)) return {log_core_(hi_(a), lo_(a), 77u), log_core_(hi_(b), lo_(b), 77u)};
  return {flog(a), flog(b)};
}
FM_NI Pair fexp2(double a, double b)
{
  // (|x| < 700: no overflow, no subnormal result)
  if ((hi_(a) & 0x7fffffffu) < 0x4085e000u && (hi_(b) & 0x7fffffffu) < 0x4085e000u) {
    uint64_t qa, qb;
    int32_t ma, mb;
    exp_parts_(a, qa, ma);
    exp_parts_(b, qb, mb);
    return {from_bits_((int64_t)(qa + ((uint64_t)(uint32_t)(ma + 1022) << 52))),
            from_bits_((int64_t)(qb + ((uint64_t)(uint32_t)(mb + 1022) << 52)))};
  }
  return {fexp(a), fexp(b)};
}

// the IEEE division, out of line (the rare fallback of the paths below)
FM_NI double div_ieee_(double a, double b) { return a / b; }

// 1/x to within 2^-62 for x = X 2^-60 in [1, 2) as a fixed-point fraction,
// Y 2^-63.
FM_HD uint64_t rcp_fixed60_(uint64_t X)
{
  const uint32_t xh = (uint32_t)(X >> 32), xl = (uint32_t)X;
  const float xf = ffrom_bits_((int32_t)(0x3f800000u | ((uint32_t)(X >> 37) & 0x7fffffu)));   // x truncated
  // y0 2^24 in [2^23, 2^24): y0 = 1 is taken one unit lower, and a seed that
  // the approximation's last unit puts below 1/2 (x next to 2) as 1/2
  const uint32_t yb = (uint32_t)fbits_(rcp_seed_(xf)), yc = yb < 0x3f7fffffu ? yb : 0x3f7fffffu;
  const uint32_t y0 = ((yc > 0x3f000000u ? yc : 0x3f000000u) & 0x7fffffu) | 0x800000u;
  // eps 2^84 = 2^84 - (x 2^60) (y0 2^24), modulo 2^64 (|eps| < 2^-21)
  const uint64_t p = (uint64_t)xl * y0 + ((uint64_t)(xh * y0) << 32);
  const int64_t e = (int64_t)(0u - p);
  const int32_t eh = (int32_t)(e >> 32);
  const int64_t w = e + (((int64_t)eh * eh) >> 20);               // eps + eps^2
  // y0 + y0 w
  const int64_t t = (int64_t)(int32_t)(w >> 32) * (int32_t)y0 + (int64_t)mulhi_((uint32_t)w, y0);   // y0 w 2^76
  return ((uint64_t)y0 << 39) + (uint64_t)(t >> 13);
}
// the same from x's 53-bit significand mh : ml
FM_HD uint64_t rcp_fixed_(uint32_t mh, uint32_t ml) { return rcp_fixed60_((((uint64_t)mh << 32) | ml) << 8); }

// The 53-bit quotient settled by its exact remainder r = a - q b (|r| far
// below 2^63, so its low 64 bits tell it): q is the rounded quotient iff
// |r| <= b / 2.
FM_HD uint64_t settle_(uint64_t q, int64_t r, uint64_t mb)
{
  const int64_t half = (int64_t)(mb >> 1);
  if (r > half) return q + 1;
  if (r < -half) return q - 1;
  return q;
}

// 1/d, correctly rounded.
FM_NI double frcp(double d)
{
  const uint32_t h = hi_(d), l = lo_(d), e = (h >> 20) & 0x7ffu;
  if (e - 1u >= 2044u) return div_ieee_(1.0, d);                  // zero, subnormal, inf, NaN; subnormal result
  const uint32_t mh = (h & 0xfffffu) | 0x100000u;
  const uint64_t m = ((uint64_t)mh << 32) | l;
  uint64_t q = (rcp_fixed_(mh, l) + 512u) >> 10;                  // 2^53 / x, in [2^52, 2^53]
  q = settle_(q, (int64_t)(0u - q * m), m);
  return from_bits_((int64_t)(q + ((uint64_t)(2044u - e) << 52) + ((uint64_t)(h & 0x80000000u) << 32)));
}

// a / b from Y = rcp_fixed_ of b's significand, correctly rounded.  ex: the
// exponent fields' difference plus 1023, in [2, 2045].
FM_HD double quot_(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, uint64_t y, uint32_t ex)
{
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  // a / b 2^62 in (2^61, 2^63): (significand of a, 64 bits) times Y, high half
  const uint32_t th = (mah << 11) | (al >> 21), tl = al << 11, yh = (uint32_t)(y >> 32), yl = (uint32_t)y;
  const uint64_t qp = (uint64_t)th * yh + mulhi_(th, yl) + mulhi_(tl, yh);
  const uint32_t lt1 = (qp >> 62) == 0 ? 1u : 0u;                 // quotient below 1: one bit more
  uint64_t q = (qp + (512u >> lt1)) >> (10u - lt1);
  const uint64_t mb = ((uint64_t)mbh << 32) | bl;
  const int64_t r = (int64_t)(((uint64_t)(al << (20u + lt1)) << 32) - q * mb);   // a 2^(52 + lt1) - q b, modulo 2^64
  q = settle_(q, r, mb);
  return from_bits_((int64_t)(q + ((uint64_t)(ex - lt1 - 1u) << 52) + ((uint64_t)((ah ^ bh) & 0x80000000u) << 32)));
}

// a / b, correctly rounded (the IEEE quotient bit for bit).
FM_NI double fdiv_rn(double a, double b)
{
  const uint32_t ah = hi_(a), al = lo_(a), bh = hi_(b), bl = lo_(b);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu, ex = ea - eb + 1023u;
  if (ea - 1u >= 2046u || eb - 1u >= 2046u || ex - 2u >= 2044u) {
    // 0 / b is common (an absent species): a signed zero
    if (((ah << 1) | al) == 0u && eb - 1u < 2046u) return from_bits_((int64_t)((uint64_t)((ah ^ bh) & 0x80000000u) << 32));
    return div_ieee_(a, b);
  }
  return quot_(ah, al, bh, bl, rcp_fixed_((bh & 0xfffffu) | 0x100000u, bl), ex);
}

FM_HD double fdiv(double a, double b) { return fdiv_rn(a, b); }

// Two quotients with one divisor.
FM_NI void fdiv_rn2(double a1, double a2, double b, double &q1, double &q2)
{
  const uint32_t ah = hi_(a1), al = lo_(a1), ch = hi_(a2), cl = lo_(a2), bh = hi_(b), bl = lo_(b);
  const uint32_t ea = (ah >> 20) & 0x7ffu, ec = (ch >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  if (ea - 1u >= 2046u || ec - 1u >= 2046u || eb - 1u >= 2046u || ea - eb + 1021u >= 2044u || ec - eb + 1021u >= 2044u) {
    q1 = fdiv_rn(a1, b);
    q2 = fdiv_rn(a2, b);
    return;
  }
  const uint64_t y = rcp_fixed_((bh & 0xfffffu) | 0x100000u, bl);
  q1 = quot_(ah, al, bh, bl, y, ea - eb + 1023u);
  q2 = quot_(ch, cl, bh, bl, y, ec - eb + 1023u);
}

// The IEEE square root and its reciprocal, out of line (the rare fallbacks).
FM_NI double sqrt_ieee_(double d) { return sqrt(d); }
FM_NI double rsqrt_ieee_(double d) { return 1.0 / sqrt(d); }

// x = X 2^-52 in [1, 4) and d = x 4^k for a positive normal d.
FM_HD void sqrt_split_(uint32_t h, uint32_t l, uint64_t &X, uint32_t &odd)
{
  odd = ~(h >> 20) & 1u;                                          // E - 1023 odd
  X = (((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | l) << odd;
}

// 1/sqrt(x) to within 2^-60 as a fixed-point fraction, Y 2^-62 in (1/2, 1].
FM_HD uint64_t rsqrt_fixed_(uint64_t X, uint32_t odd)
{
  const uint32_t xh = (uint32_t)(X >> 32), xl = (uint32_t)X;
  // x truncated to FP32: the leading 24 bits of X
  const uint32_t m = (uint32_t)(X >> (29u + odd));                // 24 bits
  const float xf = ffrom_bits_((int32_t)(((127u + odd) << 23) | (m & 0x7fffffu)));
  const uint32_t yb = (uint32_t)fbits_(rcpf_(sqrtf_(xf)));
  const uint32_t y0 = ((yb < 0x3f7fffffu ? yb : 0x3f7fffffu) & 0x7fffffu) | 0x800000u;   // y0 2^24
  // eps 2^80 = 2^80 - x y0^2 2^80 from the middle of the 102-bit product x 2^52 y0^2 2^48
  const uint64_t s = (uint64_t)y0 * y0;
  const uint32_t sl = (uint32_t)s, sh = (uint32_t)(s >> 32);
  const uint64_t p0 = (uint64_t)xl * sl;
  const uint64_t mid = (uint64_t)xl * sh + (uint64_t)xh * sl + (p0 >> 32);
  const uint64_t top = (mid >> 32) + (uint64_t)(xh * sh);
  const int64_t e = (int64_t)(0u - ((top << 44) + ((uint64_t)(uint32_t)mid << 12) + ((uint32_t)p0 >> 20)));
  const int32_t eh = (int32_t)(e >> 32);
  const int64_t w = (e >> 1) + ((3 * ((int64_t)eh * eh)) >> 19);  // eps/2 + 3 eps^2/8
  const int64_t t = (int64_t)(int32_t)(w >> 32) * (int32_t)y0 + (int64_t)mulhi_((uint32_t)w, y0);   // y0 w 2^72
  return ((uint64_t)y0 << 38) + (uint64_t)(t >> 10);
}

// 1/sqrt(d) for a positive normal d; frsqrt_ok tells.
FM_HD bool frsqrt_ok(double d) { return hi_(d) - 0x00100000u < 0x7fe00000u; }
FM_NI double frsqrt(double d)
{
  if (!frsqrt_ok(d)) return rsqrt_ieee_(d);                       // zero, subnormal, negative, inf, NaN
  const uint32_t h = hi_(d);
  uint64_t X;
  uint32_t odd;
  sqrt_split_(h, lo_(d), X, odd);
  const uint64_t q = (rsqrt_fixed_(X, odd) + 256u) >> 9;          // [2^52, 2^53]
  const uint32_t k2 = (h >> 20) - odd;                            // 2 k + 1023
  return from_bits_((int64_t)(q + ((uint64_t)(1021u + 511u - (k2 >> 1)) << 52)));
}

// sqrt(d), the IEEE result bit for bit: X times 1/sqrt(x), rounded to 53
// bits q, settled by the exact X - q^2 (nearest iff -q < X - q^2 <= q).
FM_NI double fsqrt_rn(double d)
{
  if (!frsqrt_ok(d)) return sqrt_ieee_(d);
  const uint32_t h = hi_(d);
  uint64_t X;
  uint32_t odd;
  sqrt_split_(h, lo_(d), X, odd);
  // sqrt(x) 2^62 in [2^62, 2^63): x 2^62 times Y, high half, doubled twice
  const uint64_t r = mulhi64_(X << 10, rsqrt_fixed_(X, odd)) << 2;
  uint64_t q = (r + 512u) >> 10;                                  // [2^52, 2^53]
  const int64_t rem = (int64_t)((X << 52) - q * q);               // modulo 2^64
  if (rem > (int64_t)q) ++q;
  else if (rem <= -(int64_t)q) --q;
  const uint32_t k2 = (h >> 20) - odd;
  return from_bits_((int64_t)(q + ((uint64_t)((k2 >> 1) + 511u) << 52)));
}

// atan x for |x| < 2^-7 (|x| >= 2^-30): the Taylor series, r^5 and beyond in FP32.
FM_NI double atan_small_(double x)
{
  const double x2 = mul_(x, x);
  const float f = to_f32(x2), s = fmaf_(f, fmaf_(f, 1.0f / 9.0f, -1.0f / 7.0f), 1.0f / 5.0f);
  return fma_(mul_(x2, x), fma_(x2, to_f64(s), -1.0 / 3.0), x);
}

// Arc tangent (see the header).
FM_NI double fatan(double x)
{
  const uint32_t h = hi_(x), l = lo_(x), ah = h & 0x7fffffffu, e = ah >> 20;
  if (e - 1016u >= 67u) {                                         // |x| < 2^-7 or >= 2^60, inf, NaN
    if (ah >= 0x7ff00000u && x != x) return x;
    if (e >= 1083u) return (int32_t)h < 0 ? -FM_PIO2 : FM_PIO2;
    if (e < 993u) return x;                                       // |x| < 2^-30: atan x = x (1 - x^2/3), +-0
    return atan_small_(x);
  }
  const uint32_t mh = (h & 0xfffffu) | 0x100000u;
  const bool comp = e >= 1023u;                                   // |x| >= 1: pi/2 - atan(1/|x|)
  // y = |x| or 1/|x| in (0, 1], 2^-63
  const uint64_t y = comp ? rcp_fixed_(mh, l) >> (e - 1023u) : ((((uint64_t)mh << 32) | l) << 11) >> (1023u - e);
  const uint32_t j = (uint32_t)((y + (1ull << 56)) >> 57);        // nearest multiple of 1/64
  const uint64_t c = (uint64_t)j << 57;
  // r = (y - c) / (1 + y c), |r| <= 2^-7: the magnitude 2^-69
  const bool neg = y < c;
  const uint64_t d = neg ? c - y : y - c;
  const uint64_t den = (1ull << 60) + (mulhi64_(y, c) >> 2);      // [1, 2], 2^-60
  const uint64_t q = rcp_fixed60_(den < (2ull << 60) ? den : (2ull << 60) - 1u);
  const uint64_t r = mulhi64_(d << 7, q);
  // atan r = r - r r^2 (1/3 - r^2/5 + r^4/7)
  const uint64_t r2 = sqr70_(r << 1);                             // 2^-76
  const uint32_t r46 = (uint32_t)(r2 >> 30);
  const uint32_t v = 858993459u - mulhi_(r46 >> 14, 613566757u); // (1/5 - r^2/7) 2^32
  const uint64_t w = 0x5555555555555555ull - (((uint64_t)r46 * v) >> 14);   // 2^-64
  const uint64_t ar = r - (mulhi64_(r << 1, mulhi64_(r2, w)) >> 13);        // 2^-69
  const uint64_t at = comp ? (ar + 64u) >> 7 : (ar + 16u) >> 5;   // 2^-62, 2^-64
  const AtanEntry t = atan_entry(j);
  const uint64_t res = (comp ? t.co : t.at) + ((comp != neg) ? 0u - at : at);   // (0, pi/2), 2^-62; (0, 1), 2^-64
  const uint32_t lz = (uint32_t)clz32_((uint32_t)(res >> 32));
  const uint64_t top = res << lz;
  const uint64_t m = (top >> 11) + ((uint32_t)(top >> 10) & 1u);
  return from_bits_((int64_t)(m + ((uint64_t)((comp ? 1023u : 1021u) - lz) << 52) + ((uint64_t)(h & 0x80000000u) << 32)));
}

}  // namespace fm
