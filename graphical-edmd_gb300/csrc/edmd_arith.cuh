// edmd_arith.cuh -- exact FP64 arithmetic on the integer pipe: correctly rounded
// division and square root, bit for bit the IEEE results of `a / b` and
// `sqrt(x)`, and the event calendar's repeated additions in closed form.
//
// GB300 issues one FP64 warp instruction per 64 cycles from one warp, dependent
// or not, and one per 76 cycles and SM sub-partition with all four busy; the
// compiler's FP64 division and square root are chains of about nine of them.
// Measured on GB300 (one dependent chain / 16 warps per SM, cycles per operation
// and warp, loop included): a / b 575 / 2245, div_rn 267 / 532; sqrt(x) 654 /
// 2602, sqrt_rn 280 / 497.  The event kernels are bound by FP64 issue and by the
// latency of the pair solve, so both figures count.
//
// Method: long division (and digit-by-digit square root) of the 53-bit
// significands in two digits, each estimated with a 31-bit reciprocal (root)
// that one integer Newton step refines from the FP32 approximation
// instruction.  The remainder of the two-digit result is exact modulo 2^64 and
// smaller than 2^63, so comparing it with half the divisor (the root) rounds
// to nearest.  Neither a quotient nor a root of 53-bit significands can fall
// on the midpoint of two results, so no tie rule is needed.  The FP32 seeds
// may be off by several units in their last place (2^-20 is enough), so the
// result does not depend on the approximation instruction.  Operands or
// results that are not normal numbers take the compiler's operation.
#pragma once
#include <cstdint>
#ifdef __CUDACC__
#define EDMD_HD __host__ __device__ __forceinline__
#else
#include <cstring>
#define EDMD_HD inline
#endif

namespace edmd {

EDMD_HD uint64_t f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
EDMD_HD double bits_f64(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

// bits of an FP32 approximation of 1 / x and 1 / sqrt(x); the host's take an
// error in units of the last place, to test the tolerance of the digits
#ifdef __CUDA_ARCH__
EDMD_HD uint32_t seed_rcp(uint32_t x, int) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(x)));
  return __float_as_uint(y);
}
EDMD_HD uint32_t seed_rsqrt(uint32_t x, int) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(x)));
  return __float_as_uint(y);
}
#else
EDMD_HD uint32_t seed_rcp(uint32_t x, int ulps) {
  float f;
  memcpy(&f, &x, 4);
  f = 1.0f / f;
  memcpy(&x, &f, 4);
  return x + (uint32_t)ulps;
}
EDMD_HD uint32_t seed_rsqrt(uint32_t x, int ulps) {
  float f;
  memcpy(&f, &x, 4);
  f = 1.0f / __builtin_sqrtf(f);
  memcpy(&x, &f, 4);
  return x + (uint32_t)ulps;
}
#endif

// FP32 bits of a seed of the interval (1/2, 1], which an approximation can
// leave by a few units in the last place, brought into [1/2, 1)
EDMD_HD uint32_t clamp_unit(uint32_t y) {
  y = y < 0x3f000000u ? 0x3f000000u : y;
  return y > 0x3f7fffffu ? 0x3f7fffffu : y;
}

EDMD_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// a / b for normal a, b and a normal quotient; *other is set when that does
// not hold (the value returned is then meaningless)
EDMD_HD double div_normal(double a, double b, bool* other, int seed_ulps = 0) {
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
  uint64_t ma = (ua & 0xfffffffffffffull) | (1ull << 52);
  const uint64_t mb = (ub & 0xfffffffffffffull) | (1ull << 52);
  const bool lt = ma < mb;
  if (lt) ma += ma;                                  // ma / mb in [1, 2)
  const int e = ea - eb + 1023 - (lt ? 1 : 0);
  *other = (uint32_t)(ea - 1) >= 2046u || (uint32_t)(eb - 1) >= 2046u || (uint32_t)(e - 1) >= 2046u;
  // Y = 2^32 / b, b = mb / 2^52 in [1, 2): at most 2^32 - 1, since a Newton
  // step never exceeds the value it approaches
  uint32_t y = seed_rcp(0x3f800000u | ((uint32_t)(mb >> 29) & 0x7fffffu), seed_ulps);
  y = clamp_unit(y);
  uint32_t Y = (y << 8) | 0x80000000u;
  const uint32_t B = (uint32_t)(mb >> 21);           // 2^31 b
  const int64_t er = (int64_t)((1ull << 63) - (uint64_t)Y * B);
  Y += (uint32_t)(((int64_t)(int32_t)(er >> 31) * (int64_t)(int32_t)(Y >> 1)) >> 31);
  // first digit P ~ 2^30 q (off by at most 3) and its remainder
  const uint32_t P = mul_hi((uint32_t)(ma >> 22), Y);
  const int64_t R = (int64_t)((ma << 30) - (uint64_t)P * mb);
  // second digit, rounded: Q = 2^52 q within 0.6
  const int64_t d = ((int64_t)(int32_t)(R >> 25) * (int64_t)(int32_t)(Y >> 1) + (1ll << 35)) >> 36;
  uint64_t Q = ((uint64_t)P << 22) + (uint64_t)d;
  const int64_t r = (int64_t)(((uint64_t)R << 22) - (uint64_t)d * mb);
  if (2 * r > (int64_t)mb) Q++;
  if (2 * r < -(int64_t)mb) Q--;
  return bits_f64(((ua ^ ub) & (1ull << 63)) | (((uint64_t)(uint32_t)(e - 1) << 52) + Q));
}

// sqrt(x) for positive normal x; *other is set when that does not hold
EDMD_HD double sqrt_normal(double x, bool* other, int seed_ulps = 0) {
  const uint64_t u = f64_bits(x);
  const uint32_t h = (uint32_t)(u >> 32), ex = h >> 20;
  *other = h - 0x00100000u >= 0x7fe00000u;
  const uint64_t m = (u & 0xfffffffffffffull) | (1ull << 52);
  const bool odd = !(ex & 1);                        // the unbiased exponent is odd
  const uint64_t M = odd ? m + m : m;                // v = M / 2^52 in [1, 4), s = sqrt(v)
  uint32_t y = seed_rsqrt((odd ? 0x40000000u : 0x3f800000u) | ((uint32_t)(m >> 29) & 0x7fffffu), seed_ulps);
  y = clamp_unit(y);
  uint32_t Y = (y << 8) | 0x80000000u;               // 2^32 / s
  const uint32_t V = (uint32_t)(M >> 22);            // 2^30 v
  const int64_t er = (int64_t)((1ull << 62) - (uint64_t)V * mul_hi(Y, Y));
  Y += (uint32_t)(((int64_t)(int32_t)(er >> 31) * (int64_t)(int32_t)(Y >> 1)) >> 31);
  // first digit P ~ 2^30 s and its remainder; second digit, rounded
  const uint32_t P = mul_hi(V, Y);
  const int64_t R = (int64_t)((M << 8) - (uint64_t)P * P);
  const int64_t d = ((int64_t)(int32_t)(R >> 5) * (int64_t)(int32_t)(Y >> 1) + (1ll << 34)) >> 35;
  uint64_t S = ((uint64_t)P << 22) + (uint64_t)d;
  const int64_t r = (int64_t)((M << 52) - S * S);    // 2^104 (v - S^2)
  if (r > (int64_t)S) S++;                           // v > (S + 1/2)^2
  if (r <= -(int64_t)S) S--;                         // v < (S - 1/2)^2
  const uint32_t eo = (ex + 1023u - (odd ? 1u : 0u)) >> 1;
  return bits_f64(((uint64_t)(eo - 1) << 52) + S);
}

// The serial loop's calendar walk: while P + d <= tc, P becomes fl(P + d) and k
// counts, for at most 2^24 steps.  Inside a binade of P every step but the
// first adds the same multiple of its ulp (d rounds the same way each time,
// and a tie leaves P even), so the steps up to tc or to the binade's end are
// taken at once, as integers: ~20 divisions instead of tc / d additions
// (140,000 for 10^6 disks at t = 0.7, 2.7 ms of a round that held such an event).
EDMD_HD void walk_calendar(double d, double tc, double& P, uint64_t& k) {
  int64_t left = 1 << 24;
  while (left > 0 && P + d <= tc) {
    const uint64_t p0 = f64_bits(P);
    P += d; k++; left--;
    if (left == 0 || !(P + d <= tc)) return;
    const uint64_t p1 = f64_bits(P), p2 = f64_bits(P + d), e = p1 >> 52;
    if (p0 >> 52 != e || p2 >> 52 != e || (p1 >> 63) || e == 0) continue;
    const uint64_t step = p2 - p1, tb = f64_bits(tc), end = (e + 1) << 52;
    uint64_t n = (uint64_t)left;
    if (step) {
      const uint64_t room = ((tb < end ? tb : end - 1) - p1) / step;
      if (room < n) n = room;
    }
    P = bits_f64(p1 + n * step);
    k += n;
    left -= (int64_t)n;
  }
}

#ifdef __CUDACC__
// out of line, so that the compiler does not evaluate them beside the digits
// and select
static __device__ __noinline__ double div_other(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_other(double x) { return sqrt(x); }
__device__ __forceinline__ double div_rn(double a, double b) {
  bool other;
  const double q = div_normal(a, b, &other);
  return other ? div_other(a, b) : q;
}
__device__ __forceinline__ double sqrt_rn(double x) {
  bool other;
  const double s = sqrt_normal(x, &other);
  return other ? sqrt_other(x) : s;
}
#endif

}  // namespace edmd
