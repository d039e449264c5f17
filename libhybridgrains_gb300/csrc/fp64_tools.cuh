// FP64 values through the integer pipe, and cheaper exact quotients.
//
// An FP64 instruction, conversions to and from FP64 included, takes a warp 64
// cycles of its SM sub-partition on this part, whatever the number of active
// lanes and independent or not (measured: 1.8 thread instructions per cycle and
// SM; a division 8 of them, a reciprocal 5, a square root 9), a 32-bit integer
// instruction about 1. So the count of FP64 instructions is the time of these
// kernels, and conversions, comparisons, powers of two and decisions that
// integer or FP32 arithmetic can make exactly are made there.
#pragma once

#include <stdint.h>

namespace hg {

__device__ __forceinline__ uint32_t f64_hi(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t f64_lo(double x) { return (uint32_t)__double2loint(x); }
// x is +0 or -0
__device__ __forceinline__ bool f64_zero(double x) { return ((f64_hi(x) << 1) | f64_lo(x)) == 0u; }
// a < b for values that are not negative (nor NaN)
__device__ __forceinline__ bool f64_less(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
// isfinite
__device__ __forceinline__ bool finite_bits(double x) { return (f64_hi(x) & 0x7FF00000u) != 0x7FF00000u; }
// 2 x and x / 2
static __device__ __noinline__ double scale_slow(double x, double by) { return x * by; }
__device__ __forceinline__ double twice(double x) {
  const uint32_t hi = f64_hi(x), e = (hi >> 20) & 0x7FFu;
  if (e - 1u < 2045u) return __hiloint2double((int)(hi + 0x100000u), (int)f64_lo(x));
  return f64_zero(x) ? x : scale_slow(x, 2.0);
}
__device__ __forceinline__ double halved(double x) {
  const uint32_t hi = f64_hi(x), e = (hi >> 20) & 0x7FFu;
  if (e - 2u < 2045u) return __hiloint2double((int)(hi - 0x100000u), (int)f64_lo(x));
  return f64_zero(x) ? x : scale_slow(x, 0.5);
}
// min(0, x); 0 for a NaN
__device__ __forceinline__ double min_zero(double x) {
  const uint32_t hi = f64_hi(x), lo = f64_lo(x);
  const bool nan = (hi & 0x7FFFFFFFu) > 0x7FF00000u ||
                   ((hi & 0x7FFFFFFFu) == 0x7FF00000u && lo != 0u);
  return (hi >> 31) && !nan ? x : 0.0;
}

// (float)x, rounded to nearest even, for a double in FP32's normal range;
// other values take the conversion instruction.
static __device__ __noinline__ float narrow_slow(double x) { return (float)x; }
__device__ __forceinline__ float narrow(double x) {
  const uint32_t hi = f64_hi(x), lo = f64_lo(x);
  const uint32_t e = (hi >> 20) & 0x7FFu;
  if (e - 897u < 253u) { // 2^-126 <= |x| < 2^127
    const uint64_t b = ((uint64_t)(hi & 0x7FFFFFFFu) << 32) | lo;
    const uint64_t r = b + 0x0FFFFFFFull + ((b >> 29) & 1u); // ties to even at bit 29
    return __uint_as_float(((uint32_t)(r >> 29) - (896u << 23)) | (hi & 0x80000000u));
  }
  if (((hi << 1) | lo) == 0u) return __uint_as_float(hi); // a zero keeps its sign
  return narrow_slow(x);
}
// The same truncated, for FP32 estimates.
__device__ __forceinline__ float narrow_trunc(double x) {
  const uint32_t hi = f64_hi(x), lo = f64_lo(x);
  const uint32_t e = (hi >> 20) & 0x7FFu;
  if (e - 897u < 253u)
    return __uint_as_float((((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29) |
                           (hi & 0x80000000u));
  if (((hi << 1) | lo) == 0u) return 0.0f;
  return narrow_slow(x);
}
// (double)f
static __device__ __noinline__ double widen_f32_slow(float f) { return (double)f; }
__device__ __forceinline__ double widen_f32(float f) {
  const uint32_t b = __float_as_uint(f), m = b & 0x7FFFFFFFu;
  if (m - 0x00800000u < 0x7F000000u) // normal
    return __hiloint2double((int)(((m >> 3) + (896u << 20)) | (b & 0x80000000u)), (int)(b << 29));
  if (m == 0u) return __hiloint2double((int)b, 0);
  return widen_f32_slow(f);
}
// (double)i for 0 <= i < 2^31
__device__ __forceinline__ double index_f64(int i) {
  if (i == 0) return 0.0;
  const int e = 31 - __clz(i);
  const uint64_t m = (uint64_t)(uint32_t)i << (52 - e); // leading bit at 52
  return __longlong_as_double((int64_t)(m + ((uint64_t)(e + 1022) << 52)));
}
// (int)floor(x) and (int)ceil(x); values outside [1, 2^31) take the FP64
// instructions.
static __device__ __noinline__ int floor_slow(double x) { return (int)floor(x); }
static __device__ __noinline__ int ceil_slow(double x) { return (int)ceil(x); }
__device__ __forceinline__ int floor_int(double x, bool *whole = nullptr) {
  const uint32_t hi = f64_hi(x), lo = f64_lo(x);
  const uint32_t e = (hi >> 20) - 1023u; // a sign bit gives 1025 or more
  if (e < 31u) {
    const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
    if (whole) *whole = (m << (12 + e)) == 0u;
    return (int)(m >> (52u - e));
  }
  if (whole) *whole = x == floor(x);
  return floor_slow(x);
}
__device__ __forceinline__ int ceil_int(double x) {
  const uint32_t e = (f64_hi(x) >> 20) - 1023u;
  if (e < 30u) {
    bool whole;
    const int i = floor_int(x, &whole);
    return i + (whole ? 0 : 1);
  }
  return ceil_slow(x);
}

// Quotients by one divisor. With y = 1 / b rounded to nearest, the multiply
// q = a y followed by the residual correction q + (a - q b) y in two FMAs
// gives a / b rounded to nearest (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990), three FP64
// instructions in place of a division's eight. Operands near the ends of the
// exponent range clear ok; the caller then takes true divisions, one branch for
// a group of quotients.
struct Divisor {
  double b, y;
  bool ok;
};
// y: 1 / b rounded to nearest
__device__ __forceinline__ Divisor divisor(double b, double y) {
  const uint32_t e = (f64_hi(b) >> 20) & 0x7FFu;
  return {b, y, e - 823u <= 400u};
}
__device__ __forceinline__ Divisor divisor(double b) { return divisor(b, 1.0 / b); }
__device__ __forceinline__ double quot(double a, const Divisor &d, bool &ok) {
  const uint32_t e = (f64_hi(a) >> 20) & 0x7FFu;
  ok = ok && (e - 300u <= 1400u || f64_zero(a));
  const double q = a * d.y;
  return fma(fma(-q, d.b, a), d.y, q); // (a zero comes out as +0)
}
static __device__ __noinline__ double divide(double a, double b) { return a / b; }
// a single quotient
__device__ __forceinline__ double quot(double a, const Divisor &d) {
  bool ok = d.ok;
  const double z = quot(a, d, ok);
  return ok ? z : divide(a, d.b);
}
// SAFE: by division
template <bool SAFE>
__device__ __forceinline__ double quot_or(double a, const Divisor &d, bool &ok) {
  return SAFE ? a / d.b : quot(a, d, ok);
}

// sqrt(a) and its reciprocal by Goldschmidt's iteration (R. Goldschmidt, 1964;
// P. Markstein, "Software division and square root using Goldschmidt's
// algorithms", 2004) from an FP32 estimate: one iteration to about 2^-43 and a
// residual correction of each, which leaves both rounded to nearest but for
// one argument in 2^32 or so (then within one unit). 8 FP64 instructions (6
// where the reciprocal is not used) in place of 14 (9).
static __device__ __noinline__ double2 root_slow(double a) {
  const double g = sqrt(a);
  return make_double2(g, 1.0 / g);
}
__device__ __forceinline__ double2 root(double a) {
  const uint32_t e = (f64_hi(a) >> 20) - 898u; // a sign bit makes it large
  if (e > 250u) return root_slow(a);
  const double y0 = widen_f32(rsqrtf(narrow_trunc(a)));
  double g = a * y0, h = halved(y0);
  const double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  g = fma(fma(-g, g, a), h, g);
  const double y = twice(h);
  return make_double2(g, fma(y, fma(-g, y, 1.0), y));
}

} // namespace hg
