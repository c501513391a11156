// ice3gb_device.cuh — device-side helpers shared by the ICE3 kernels.
//
// Layout: every 3-D field is [nk][nij] FP64 (ij fastest), 2-D fields [nij].
// The constants table (Ice3gbConstants, ~1.5 KB) is passed by value as a
// __grid_constant__ kernel parameter, so every lane reads it from the
// constant bank with no global-memory traffic.
#pragma once

#include <stdint.h>
#if defined(__CUDACC__)
#include <cuda_runtime.h>
#else
#include <cmath>
using std::exp; using std::log; using std::fmin; using std::fmax; using std::sqrt; using std::fabs;
using std::signbit;
#endif

#include "../../include/ice3gb.h"
#include "fastmath.cuh"

typedef Ice3gbConstants Cst;

#if defined(__CUDACC__)
#define ICE3_HD __host__ __device__ __forceinline__
#else
#define ICE3_HD inline
#endif

ICE3_HD double sq(double x) { return x * x; }
// Separately rounded multiply and add (never fused into an FMA).
ICE3_HD double mul_rn(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  volatile double p = a * b;
  return p;
#endif
}
ICE3_HD double add_rn(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  volatile double p = a + b;
  return p;
#endif
}
// The bit pattern of x through an inline-assembly move, which the compiler
// cannot see through: a test that equals an FP64 comparison (x == 0, x != 0)
// would otherwise be turned back into one, on the FP64 pipe.
ICE3_HD uint64_t opaque_bits(double x)
{
#if defined(__CUDA_ARCH__)
  unsigned long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
#else
  return (uint64_t)fm::bits_(x);
#endif
}
// Comparisons and clamps on the IEEE bit patterns.  On GB300 an FP64 compare
// (and so fmin/fmax) issues on the FP64 pipe at the FP64 FMA rate, while the
// same test on the 64-bit pattern runs on the integer pipe at ~30x the rate.
// Ordering key: for non-NaN doubles the signed 64-bit integer
// (sign ? -|bits| : bits) orders like the values, with -0 and +0 equal as
// IEEE compares them.  The plain versions below do not handle NaN operands
// (their callers see finite values by construction); nmin/nmax do.
ICE3_HD int64_t dkey(double x)
{
  const int64_t b = fm::bits_(x);
  return b < 0 ? -(b & 0x7fffffffffffffffLL) : b;
}
ICE3_HD bool isnan_(double a) { return (fm::bits_(a) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL; }

// NaN-propagating minimum/maximum/clip, as numpy's minimum/maximum/clip
// (the reference JAX lets NaN through on degenerate inputs, e.g. a negative
// vapour source with no mass flux, stencils/ice_adjust.py:293-296); CUDA's
// fmin/fmax would return the other operand instead.  Same results as
// (a < b || a != a) ? a : b, evaluated on the integer pipe.
ICE3_HD double nmin(double a, double b) { return (isnan_(a) || (!isnan_(b) && dkey(a) < dkey(b))) ? a : b; }
ICE3_HD double nmax(double a, double b) { return (isnan_(a) || (!isnan_(b) && dkey(a) > dkey(b))) ? a : b; }
ICE3_HD double nclip01(double x) { return nmin(nmax(x, 0.0), 1.0); }
// IEEE a > b / a >= b (false when either is NaN), on the integer pipe.
ICE3_HD bool fgt(double a, double b) { return !isnan_(a) && !isnan_(b) && dkey(a) > dkey(b); }
ICE3_HD bool fge(double a, double b) { return !isnan_(a) && !isnan_(b) && dkey(a) >= dkey(b); }
ICE3_HD bool gtd(double a, double b) { return dkey(a) > dkey(b); }        // a > b
ICE3_HD bool ltd(double a, double b) { return dkey(a) < dkey(b); }        // a < b
// a > b for a threshold b >= +0 (a of any sign): the raw patterns suffice.
ICE3_HD bool gtp(double a, double b) { return fm::bits_(a) > fm::bits_(b); }
// a < b for a >= +0 (b of any sign >= +0).
ICE3_HD bool ltp(double a, double b) { return fm::bits_(a) < fm::bits_(b); }
ICE3_HD bool pos(double a) { return fm::bits_(a) > 0; }                   // a > 0
ICE3_HD double pmax0(double a) { return pos(a) ? a : 0.0; }               // fmax(0, a)
ICE3_HD double dmax(double a, double b) { return gtd(a, b) ? a : b; }
ICE3_HD double dmin(double a, double b) { return gtd(a, b) ? b : a; }
// a == +-0.
ICE3_HD bool zerod_(double a) { return (opaque_bits(a) << 1) == 0; }
// x < 0 (not -0), on the bit pattern.
ICE3_HD bool negd(double x) { return fm::bits_(x) < 0 && fm::bits_(x) != INT64_MIN; }
// |a| > b for b >= +0.
ICE3_HD bool abs_gtp(double a, double b) { return (fm::bits_(a) & 0x7fffffffffffffffLL) > fm::bits_(b); }
// a != 0 (nor -0), on the bit pattern.
ICE3_HD bool nz(double a) { return (opaque_bits(a) << 1) != 0; }
// neither infinite nor NaN.
ICE3_HD bool finite_(double a) { return (fm::hi_(a) & 0x7fffffffu) < 0x7ff00000u; }
// True on every lane when the predicate holds on some active lane of the warp:
// a block of arithmetic that is exact when skipped on lanes whose inputs are
// zero runs for the warp or for none of it (the host build: the lane alone).
ICE3_HD bool warp_any(bool p)
{
#if defined(__CUDA_ARCH__)
  return __any_sync(__activemask(), p);
#else
  return p;
#endif
}

// num / den in FP32, to within 2^-20 relative (both truncated to FP32, the
// hardware's reciprocal); exact in sign.  0 where either is outside FP32's
// normal range.  Used to skip an IEEE division whose result cannot change a
// min / max, without an FP64 operation.
ICE3_HD float quot_est(double num, double den)
{
  const uint32_t en = (fm::hi_(num) >> 20) & 0x7ffu, ed = (fm::hi_(den) >> 20) & 0x7ffu;
  if (en - 899u >= 250u || ed - 899u >= 250u) return 0.0f;
  return fm::mulf_(fm::to_f32(num), fm::rcp_seed_(fm::to_f32(den)));
}
// True only if the quotient that est estimates (quot_est) is above bound
// for certain: above the truncated bound by 2^-17, the bound positive and within
// 2^-126 .. 2^126 (a smaller one truncates to 0, and the 0 that stands for no
// estimate is above a negative one; a caller then forms the quotient).
ICE3_HD bool est_above(float est, double bound)
{
  if ((fm::hi_(bound) >> 20) - 897u >= 252u) return false;
  const float b = fm::to_f32(bound);
  return est > fm::fmaf_(b, 0x1p-17f, b);
}
ICE3_HD bool quot_above(double num, double den, double bound) { return est_above(quot_est(num, den), bound); }

// x**a evaluated as exp(a*log(x)) with the FP64-lean exp/log of
// fastmath.cuh.  For the exponents of the scheme (|a*log x| < 60) this stays
// within ~1e-14 relative of pow(), well inside the 1e-10 parity bar, at a
// fraction of the FP64 instructions; callers raising one base to several
// powers pass a shared log.
ICE3_HD double powl_(double logx, double a) { return fm::fexp(a * logx); }

// TIWMX saturation tables of OCND2 (micro/modd_tiwmx.F90, filled by
// micro/mode_ini_tiwmx.F90 from micro/mode_tiwmx_fun.F90) at T = j/100 K,
// j = 13200..37316, stored one after the other: ESTABW, ESTABI (the ice
// formula at and below 273.15 K, the water one above), A2TAB (AA2), BB3TAB
// (BB3), AM3TAB (AM3, 0 above 273.15 K), REDINTAB (REDIN).
constexpr int kTiwmxStart = 13200, kTiwmxStop = 37316, kTiwmxN = kTiwmxStop - kTiwmxStart + 1;
enum { TW_ESW = 0, TW_ESI, TW_A2, TW_BB3, TW_AM3, TW_REDIN, TW_N };

// TAB(NINT(100 T)) (micro/mode_tiwmx.F90), NINT rounding half away from
// zero; the index is clamped to the table.
ICE3_HD double tiwmx_at(const double *tab, double t)
{
  long j = (long)round(100.0 * t);
  j = j < kTiwmxStart ? kTiwmxStart : (j > kTiwmxStop ? kTiwmxStop : j);
#if defined(__CUDA_ARCH__)
  return __ldg(tab + (j - kTiwmxStart));
#else
  return tab[j - kTiwmxStart];
#endif
}

#if defined(__CUDACC__)
// p mod nij, in 32 bits where p allows it (a 64-bit remainder is a call of
// ~100 instructions).
__device__ __forceinline__ long column_of(long p, int nij)
{
  return p <= 0xffffffffL ? (long)((unsigned)p % (unsigned)nij) : p % nij;
}
__device__ __forceinline__ double ld1(const double *p, long i) { return __ldg(p + i); }
#endif
