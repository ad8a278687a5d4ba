// FP64 reciprocals, square roots and comparisons for kernels bound by the
// FP64 pipe (sm_103a).
//
// GB300 executes two FP64 lanes per SM and clock, so one FP64 warp instruction
// takes the pipe as long as 64 issue slots of the other pipes.  1.0 / x,
// sqrt(x) and rsqrt(x) cost seven to ten FP64 instructions each.  Here the
// seed of the Newton iteration is brought to about 46 bits on the FP32 and
// integer pipes, so that ONE Newton step in FP64 finishes it:
//   rcp   2 FP64 instructions   e = 1 - x r,  r + r e
//   sqrt  3                     s = x y, e = x - s s, s + (y/2) e
//   rsqrt 3                     e = 1 - (x y) y, y + (y/2) e
// The seed: the significand of x as a float h (top 24 bits) and its rest l;
// r0 the hardware's approximate float reciprocal (root) of h; the residual
// e = 1 - (h + l) r0 (1 - (h + l) r0^2) formed with FMAs, exact to about 2^-47,
// and r0 (1 + e + e^2) (r0 (1 + e/2 + 3 e^2/8)), the Newton-Raphson series
// with its second-order term.  The correction is added to the double's bit
// pattern as an integer, the exponent likewise, so no FP64 instruction and no
// double conversion is spent on the seed.
//
// Measured in the Roe-MUSCL step on 134^3 cells (ten roots and three reciprocals a
// face): part of the fall from 12.3 to 9.3 ms a step described in roe_flux.cuh.
//
// The errors after the FP64 step: rcp and sqrt within 0.51 ulp, rsqrt
// within 1 ulp (tests/test_gpu_fd64.py), as the functions they stand for.
// Arguments outside the range of the seed (zero, subnormal, infinite, NaN, the
// exponents near them, negative for the roots) take those functions.
#pragma once
#include <cuda_runtime.h>

namespace cans {
namespace fd {

static __device__ __noinline__ double rcp_any(double x) { return 1.0 / x; }
static __device__ __noinline__ double sqrt_any(double x) { return x == 0.0 ? x : sqrt(x); }
static __device__ __noinline__ double rsqrt_any(double x) { return rsqrt(x); }

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// r0 + k 2^-51 as a double, r0 in [1/2, 1), with its exponent field moved by
// (hadj - 0x3fe00000) >> 20
__device__ __forceinline__ double seed_double(float r0, int k, unsigned hadj) {
  const unsigned u = __float_as_uint(r0);
  const unsigned long long b =
      ((unsigned long long)(((u >> 3) & 0xfffffu) + hadj) << 32) | (u << 29);
  return __longlong_as_double((long long)(b + (unsigned long long)((long long)k << 2)));
}

// 1 / x
__device__ __forceinline__ double rcp(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (((hi >> 20) & 0x7ffu) - 2u > 2042u) return rcp_any(x);
  const float h = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);
  const float l = __fmul_rn(__uint2float_rn(lo & 0x1fffffffu), 0x1p-52f);
  // within [1/2, 1 - 2^-24], so that the integer correction stays in one binade
  const float r0 = fmaxf(fminf(rcp_approx(h), 0x1.fffffep-1f), 0.5f);
  const float e = __fmaf_rn(-l, r0, __fmaf_rn(-h, r0, 1.0f));
  const int k = __float2int_rn(__fmul_rn(__fmul_rn(r0, 0x1p51f), __fmaf_rn(e, e, e)));
  // r0 stands for 1/h: the exponent field 1022 + (1023 - E), and the sign
  const unsigned adj = (0x7fd00000u - (hi & 0x7ff00000u)) | (hi & 0x80000000u);
  const double r = seed_double(r0, k, adj);
  return fma(r, fma(-x, r, 1.0), r);
}

// the seed of 1 / sqrt(x) for a positive normal x
__device__ __forceinline__ double rsqrt_seed(unsigned hi, unsigned lo) {
  // x = (h + l) 4^q with h in [1, 4): p = 1 where the exponent is odd
  const unsigned E = hi >> 20, p = (E & 1u) ^ 1u;
  const float h =
      __uint_as_float(((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u) + (p << 23));
  const float l = __fmul_rn(__uint2float_rn(lo & 0x1fffffffu),
                            __uint_as_float((75u + p) << 23));  // 2^-52 2^p
  const float r0 = fmaxf(fminf(rsqrt_approx(h), 0x1.fffffep-1f), 0.5f);
  const float t = __fmul_rn(r0, r0), tl = __fmaf_rn(r0, r0, -t);
  const float e = __fmaf_rn(-l, t, __fmaf_rn(-h, tl, __fmaf_rn(-h, t, 1.0f)));
  const int k = __float2int_rn(
      __fmul_rn(__fmul_rn(r0, 0x1p51f), __fmul_rn(e, __fmaf_rn(0.375f, e, 0.5f))));
  // exponent field 1022 - (E - 1023 - p) / 2
  const unsigned adj = (1022u + ((1023u + p - E) >> 1)) << 20;
  return seed_double(r0, k, adj & 0x7ff00000u);
}
// positive, exponent field 128 .. 2046: far enough from the smallest numbers
// that the residual x - s s (2^-105 of x in its last bit) loses nothing
__device__ __forceinline__ bool root_range(unsigned hi) {
  return hi - 0x08000000u < 0x77f00000u;
}
__device__ __forceinline__ double half_of(double y) {  // y / 2 on the integer pipe
  return __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
}

// sqrt(x)
__device__ __forceinline__ double sqrt_(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (!root_range(hi)) return sqrt_any(x);
  const double y = rsqrt_seed(hi, lo);
  const double s = x * y;
  return fma(half_of(y), fma(-s, s, x), s);
}
// 1 / sqrt(x)
__device__ __forceinline__ double rsqrt_(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (!root_range(hi)) return rsqrt_any(x);
  const double y = rsqrt_seed(hi, lo);
  return fma(half_of(y), fma(-(x * y), y, 1.0), y);
}
// both, from one seed
__device__ __forceinline__ void sqrt_rsqrt(double x, double &s, double &r) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (!root_range(hi)) {
    s = sqrt_any(x);
    r = rsqrt_any(x);
    return;
  }
  const double y = rsqrt_seed(hi, lo);
  const double s0 = x * y, hy = half_of(y);
  s = fma(hy, fma(-s0, s0, x), s0);
  r = fma(hy, fma(-s0, y, 1.0), y);
}

// Comparisons of doubles on the integer pipe.  The bit patterns of doubles of
// one sign order like integers; key() extends the order to both signs (-0 just
// below +0, NaNs beyond the infinities).
__device__ __forceinline__ long long key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
__device__ __forceinline__ bool lt(double a, double b) { return key(a) < key(b); }
__device__ __forceinline__ double max_(double a, double b) { return lt(b, a) ? a : b; }
__device__ __forceinline__ double min_(double a, double b) { return lt(a, b) ? a : b; }
__device__ __forceinline__ bool is_nan(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
// of two values that are not negative
__device__ __forceinline__ bool ltp(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ double maxp(double a, double b) { return ltp(b, a) ? a : b; }
__device__ __forceinline__ double minp(double a, double b) { return ltp(a, b) ? a : b; }
// max(0, a): a NaN with its sign clear stays
__device__ __forceinline__ double pos_part(double a) { return __double2hiint(a) < 0 ? 0.0 : a; }
// |b| or -|b| with the sign of s flipped in: b * sign(1, s)
__device__ __forceinline__ double mul_sign(double b, double s) {
  return __hiloint2double(__double2hiint(b) ^ (__double2hiint(s) & (int)0x80000000),
                          __double2loint(b));
}
__device__ __forceinline__ double abs_(double x) {
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

}  // namespace fd
}  // namespace cans
