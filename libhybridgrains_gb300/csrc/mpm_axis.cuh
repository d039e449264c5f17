// 1-D factors of the FP64 bases over the few nodes a point or grain touches,
// in as few FP64 instructions as keep their accuracy (fp64_tools.cuh says why).
// Offsets x - x_i, which cancel, are formed with the reference's operations
// one by one; included by translation units compiled with --fmad=false. SAFE
// forms use true divisions and are for the rare caller whose quotients did not
// pass quot()'s check.
#pragma once

#include "fp64_tools.cuh"

namespace hg {

constexpr int STENCIL_AXIS = 4; // nodes per axis held; wider stencils go node by node

// x with its sign flipped where neg is the sign bit (0 or 0x80000000)
__device__ __forceinline__ double flip(double x, uint32_t neg) {
  return __hiloint2double((int)(f64_hi(x) ^ neg), (int)f64_lo(x));
}
__device__ __forceinline__ double magnitude(double x) {
  return __hiloint2double((int)(f64_hi(x) & 0x7FFFFFFFu), (int)f64_lo(x));
}
__device__ __forceinline__ double node_f64(int i) { return i >= 0 ? index_f64(i) : (double)i; }

// floor and ceil of x / h to the bit: from x times the reciprocal unless that
// is within 2^-29 of a whole number (or beyond 2^20)
struct Cells {
  int lo, hi;
};
template <bool SAFE>
__device__ __forceinline__ Cells cells(double x, const Divisor &H, bool &ok) {
  const double u = x * H.y;
  const uint32_t e = (f64_hi(u) >> 20) - 1023u;
  const uint64_t m = ((uint64_t)((f64_hi(u) & 0xFFFFFu) | 0x100000u) << 32) | f64_lo(u);
  if (!SAFE && e < 20u) {
    const uint64_t frac = m << (12u + e);
    const int c = (int)(m >> (52u - e));
    if (frac + (1ull << 35) >= (1ull << 36)) return {c, c + 1};
  }
  const double z = quot_or<SAFE>(x, H, ok);
  return {floor_int(z), ceil_int(z)};
}

template <int BASIS> struct Axis;

// LinearBasisFunctions.cpp:6-22, 53-59, 81-136: nodes i0, i0 + 1 at offsets
// d = ((x - h i) - g) / h; w = 1 - |d|, dw/dx = -sign(d) / h.
template <> struct Axis<HG_BASIS_LINEAR> {
  static constexpr uint32_t NO_SLOPE = 1u; // derivative 0 (else the sign bit of it)
  int i0, n;
  double w[2], v[2]; // weight, weight / h
  uint32_t sg[2];
  // the reference's node range
  template <bool SAFE>
  __device__ __forceinline__ void range(double x, double, double g, const Divisor &H, bool &ok) {
    i0 = cells<SAFE>(x - g, H, ok).lo;
    n = 2;
  }
  template <bool SLOPES, bool SAFE>
  __device__ __forceinline__ void factors(double x, double g, const Divisor &H, bool &ok) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double d = quot_or<SAFE>((x - H.b * node_f64(i0 + k)) - g, H, ok);
      const double a = magnitude(d);
      const bool in = f64_less(a, 1.0);
      w[k] = in ? 1.0 - a : 0.0;
      if (SLOPES) {
        v[k] = w[k] * H.y;
        // -1 for d >= 0 (a zero of either sign too), 1 for d < 0, 0 beyond 1
        sg[k] = f64_less(1.0, a) ? NO_SLOPE
                                 : (f64_hi(d) >> 31 && !f64_zero(d) ? 0u : 0x80000000u);
      }
    }
  }
};

// uGIMPLinearBasisFunctions.cpp:6-42, 71-94, 110-156, for a half-width L and
// a = |x - x_i|:
//   a >= h + L      0
//   a >= h - L      (h + L - a)^2 / 2h,         slope (h + L - a) / h
//   a >= L          2 L (1 - a / h),            slope 2 L / h
//   else            2 L - (L^2 + a^2) / h,      slope 2 a / h
// The cases are selected, not branched on (an FP64 instruction costs a warp the
// same for one lane as for 32), over one quotient r = m / h with m = h + L - a
// in the first and a in the others: r m / 2, 2 L (1 - r), (2 L - L^2 / h) - a r.
// (m is exact where it is small, so products with 1 / h in place of quotients
// keep small weights' relative accuracy.)
struct Extent { // of a point, the same for both axes
  double L, wide, inner, two, two_h, rest;
  __device__ __forceinline__ void set(double l, const Divisor &H) {
    L = l;
    wide = H.b + l;
    inner = H.b - l;
    two = twice(l);
    two_h = two * H.y;
    rest = fma(-(l * l), H.y, two);
  }
};
template <> struct Axis<HG_BASIS_UGIMP> {
  int i0, n;
  double w[STENCIL_AXIS], d[STENCIL_AXIS];
  // The reference's node range to the bit: a node that an extent touches up to
  // rounding has a weight near 1e-33 or none, and any velocity.
  template <bool SAFE>
  __device__ __forceinline__ void range(double x, double L, double g, const Divisor &H, bool &ok) {
    i0 = cells<SAFE>((x - L) - g, H, ok).lo;
    n = cells<SAFE>((x + L) - g, H, ok).hi - i0 + 1;
  }
  template <bool SLOPES>
  __device__ __forceinline__ void factors(double x, const Extent &E, double g, const Divisor &H) {
#pragma unroll
    for (int k = 0; k < STENCIL_AXIS; ++k) {
      w[k] = 0.0;
      d[k] = 0.0;
      if (k == 3 && n <= 3) continue; // (three nodes unless the extent is above h)
      const double s = x - (H.b * node_f64(i0 + k) + g);
      const double a = magnitude(s);
      const bool in = k < n && f64_less(a, E.wide);
      const bool edge = !f64_less(a, E.inner), mid = !edge && !f64_less(a, E.L);
      const double m = edge ? E.wide - a : a;
      const double r = m * H.y;
      const double z = edge ? r : fma(mid ? -1.0 : -a, r, mid ? 1.0 : E.rest);
      w[k] = in ? (edge ? halved(m) : (mid ? E.two : 1.0)) * z : 0.0;
      if (SLOPES) // (at a zero offset the slope is 0 either way)
        d[k] = in ? flip(mid ? E.two_h : (edge ? r : twice(r)), ~f64_hi(s) & 0x80000000u) : 0.0;
    }
  }
};

} // namespace hg
