// FP64 reciprocal and square root seeded on the FP32 pipes.  GB300 issues 2
// FP64 instructions per clock per SM against 128 FP32 and 64 integer ones,
// and every FP64 kernel of the path keeps that pipe 80-93 % busy, so what
// counts is FP64 instructions, not operations.  Here an FP32 hardware
// approximation y0 gives a seed with relative error e below 2^-21, and one
// third-order step of the binomial series, with the residual e formed by a
// fused multiply-add, leaves an error of order e^3 < 2^-63 before the last
// rounding:
//   1/x:       e = 1 - x y0,     1/x       = y0 (1 + e + e^2 + O(e^3))
//   x^(-1/2):  e = 1 - x y0^2,   x^(-1/2)  = y0 (1 + e/2 + 3 e^2/8 + O(e^3))
// (the series of (1 - e)^-1 and (1 - e)^-1/2; with h = x y0 the second also
// gives sqrt(x) = h (1 + e/2 + 3 e^2/8)).  A reciprocal costs 3 FP64
// instructions, a root 6 and a root with its reciprocal 6; the conversions to and from the seed run on the integer pipes.
// Operands outside 2^-100 .. 2^100 (zero, negative, infinite and NaN among
// them) take the plain operators.
#pragma once

#include <cuda_runtime.h>

namespace pcfd {

// positive with a binary exponent of -100 .. 99: one unsigned compare on the
// high word
constexpr unsigned kSeedSpan = 200u << 20;
__device__ __forceinline__ unsigned seed_offset(double x) { return (unsigned)(__double2hiint(x) - ((1023 - 100) << 20)); }
__device__ __forceinline__ bool seed_range(double x) { return seed_offset(x) < kSeedSpan; }
// |v| without the sign bit
__device__ __forceinline__ double abs_bits(double v) {
  return __hiloint2double(__double2hiint(v) & 0x7fffffff, __double2loint(v));
}
// FP32 value of a double in seed_range (truncated) and back (exact)
__device__ __forceinline__ float seed_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x) - ((1023u - 127u) << 20);
  return __uint_as_float(__funnelshift_l((unsigned)__double2loint(x), hi, 3));
}
__device__ __forceinline__ double seed_f64(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b >> 3) + ((1023u - 127u) << 20)), (int)(b << 29));
}
__device__ __forceinline__ float rcp_f32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_f32(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float sqrt_f32(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// FP32 estimate of a double of any sign and size (relative error below 2^-22
// in FP32's normal range, 0 below it, NaN above it and for infinities)
__device__ __forceinline__ float est_f32(double x) {
  const int hi = __double2hiint(x);
  const int m = (hi & 0x7fffffff) - ((1023 - 127) << 20);
  const unsigned b = m < (1 << 20)      ? 0u
                     : m >= (255 << 20) ? 0x7fffffffu
                                        : __funnelshift_l((unsigned)__double2loint(x), (unsigned)m, 3);
  return __uint_as_float(b | ((unsigned)hi & 0x80000000u));
}

// an FP32 value as a double, exactly, on the integer pipes (the conversion
// instruction runs on the FP64 pipe); zero, subnormal, infinite and NaN
// values take the conversion
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u) return m == 0u ? __hiloint2double((int)b, 0) : (double)f;
  return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + ((1023u - 127u) << 20))), (int)(b << 29));
}

// 1 / x: within 0.5 ulp + 2^-10 ulp
__device__ __forceinline__ double recip(double x) {
  if (!seed_range(x)) return 1.0 / x;
  const double y0 = seed_f64(rcp_f32(seed_f32(x)));
  const double e = fma(-x, y0, 1.0);
  return fma(y0, fma(e, e, e), y0);
}

// 1 / x for a density whose product with 1 / x stands for 1 in what follows:
// NaN instead of 0 for an infinite one
__device__ __forceinline__ double recip_finite(double x) {
  return seed_range(x) ? recip(x) : 1.0 / x + (x - x);
}

// a / b within 0.5 ulp + 2^-20 ulp: the quotient's residual formed exactly.
// Its sign is such that a zero's quotient keeps its own (q - (b q - a) / b).
__device__ __forceinline__ double quot(double a, double b) {
  const double ab = abs_bits(b);
  if (!seed_range(ab) || !(seed_range(abs_bits(a)) || abs_bits(a) == 0.0)) return a / b;
  const double r = recip(ab);
  const double q = a * r;
  const double v = fma(-fma(ab, q, -a), r, q);
  return __double2hiint(b) < 0 ? -v : v;
}

// Quotients by one denominator: its reciprocal is shared and each quotient
// corrected by its residual, 3 FP64 instructions apiece (rounded as quot's)
struct Quot64 {
  double b, r;
  bool ok;
  __device__ __forceinline__ explicit Quot64(double x) : b(x), r(0.0), ok(seed_range(x)) {
    if (ok) r = recip(x);
  }
  __device__ __forceinline__ double of(double a) const {
    if (!ok || !(abs_bits(a) == 0.0 || seed_range(abs_bits(a)))) return a / b;
    const double q = a * r;
    return fma(-fma(b, q, -a), r, q);
  }
};

// sqrt(x) and *inv = 1 / sqrt(x), each within 1 ulp (of the seeded range)
__device__ __forceinline__ double sqrt_inv(double x, double* inv) {
  if (!seed_range(x)) {
    const double s = ::sqrt(x);
    *inv = 1.0 / s;
    return s;
  }
  const double y0 = seed_f64(rsqrt_f32(seed_f32(x)));
  const double h = x * y0;
  const double e = fma(-h, y0, 1.0);
  const double t = e * fma(e, 0.375, 0.5);
  *inv = fma(y0, t, y0);
  return fma(h, t, h);
}
// sqrt(x) alone, within 0.5 ulp + 2^-20 ulp: one coupled Newton step for the
// root and half its reciprocal (relative error 2^-41), then the residual
// x - s^2 formed exactly
__device__ __forceinline__ double root(double x) {
  if (!seed_range(x)) return ::sqrt(x);
  const float r0 = rsqrt_f32(seed_f32(x));
  const double y0 = seed_f64(r0), g0 = seed_f64(0.5f * r0);
  const double h = x * y0;
  const double e = fma(-h, g0, 0.5);
  const double s = fma(h, e, h), g = fma(g0, e, g0);
  return fma(fma(-s, s, x), g, s);
}

// Comparisons of doubles on the integer pipes.
// a key that orders doubles as their values (NaN beyond the infinities)
__device__ __forceinline__ long long order_key(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
// the double of a key
__device__ __forceinline__ double key_value(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
__device__ __forceinline__ bool key_gt(double a, double b) { return order_key(a) > order_key(b); }
// infinite or NaN
__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

}  // namespace pcfd
