// The DEM broadphase's bins: shared by the kernels that move the bodies last in
// a step (the DEM's integration, the hybrid step's transfer) and bin them for
// the next step's pair search. Included by translation units compiled with
// --fmad=false.
#pragma once

#include "fp64_tools.cuh"

namespace hg {

// Bucket of a cell: blocks of 4 x 4 cells are hashed, their cells lie side by
// side, so that a neighbourhood's heads share a few cache lines. The table has
// at least 16 buckets.
__device__ __forceinline__ uint32_t cell_bucket(int cx, int cy, uint32_t mask) {
  const uint32_t block = (uint32_t)(cx >> 2) * 73856093u ^ (uint32_t)(cy >> 2) * 19349663u;
  return (block << 4 | (uint32_t)(cy & 3) << 2 | (uint32_t)(cx & 3)) & mask;
}

// Per body, for the pair search: the home cell (the cell of its centre) and,
// in FP32, the offset of the centre from the home cell's corner and the
// radius, with the fixed flag and the active static planes
// (StaticPlaneCircleConstraint::isActive, StaticPlaneCircleConstraint.cpp:
// 12-17) as bits; active static drums take the bits after the planes'. Per
// candidate pair the search needs FP32 only, except for the exact tests of
// the pairs that survive the FP32 filter.
//
// The bodies of a hash bucket are a linked list (head per bucket, the next
// body in the record), built with one exchange per body: the search needs no
// bucket counts, so no scan and no second pass over the bodies. The order of
// a list does not matter: the emission pass sorts what the search finds.
// (Buckets of a sector with their first six bodies inline instead: the search
// of 10,000 disks at 2.8 contacts each 10.8 against 12.1 us, of a million 169
// against 97 us; not kept.)
struct BinArgs {
  int64_t n;
  double H, invH;
  uint32_t mask;
  int nplanes;
  double px[HG_MAX_PLANES][2], pn[HG_MAX_PLANES][2];
  float pxf[HG_MAX_PLANES][2], pnf[HG_MAX_PLANES][2];
  int ndrums;
  double dx[HG_MAX_DRUMS][2], dr[HG_MAX_DRUMS];
  const double *r;
  const uint8_t *fixed;
  float4 *rec; // 2 per body: (offset x, offset y, radius, flags), (home cell x, y, next, -)
  int32_t *heads; // per bucket, -1: none
  unsigned long long *pc; // contact counts by kind (PC_*)
  int32_t *in_count;      // contacts in which the body is the second
  int32_t *tiles;         // sums of the four counts per tile, or nullptr
  int tile_shift;
};

enum : uint32_t { REL_FIXED = 1u, REL_PLANE0 = 2u };
static_assert(1 + HG_MAX_PLANES + HG_MAX_DRUMS <= 32, "static-object bits of the body record");

constexpr int MAXP = 32; // partner list capacity per body, kind and step

// Contact counts of a first body in one word: static objects in bits 0-7,
// circle-circle in 8-35, kinematic in 36-63. The search adds to it with one
// atomic per contact, which also gives the partner's slot. The last two are
// the partners found; at most MAXP of each kind are kept.
constexpr int PC_CC = 8, PC_KIN = 36;
__device__ __forceinline__ int pc_static(unsigned long long p) { return (int)(p & 0xFFu); }
__device__ __forceinline__ int pc_found_cc(unsigned long long p) {
  return (int)((p >> PC_CC) & 0xFFFFFFFu);
}
__device__ __forceinline__ int pc_found_kin(unsigned long long p) { return (int)(p >> PC_KIN); }
__device__ __forceinline__ int pc_cc(unsigned long long p) { return min(pc_found_cc(p), MAXP); }
__device__ __forceinline__ int pc_kin(unsigned long long p) { return min(pc_found_kin(p), MAXP); }

// Cell floor(x / H) of a coordinate and the FP32 offset from the cell's lower
// edge. x / H is formed in fixed point with 24 fraction bits by one FP64 FMA
// (adding 3 * 2^27 leaves an ulp of 2^-24), so the split is integer work; the
// binning only has to be the same for every body and monotone. Rounding moves
// a coordinate by at most 2^-25 cells, and contacts are at most
// H / (1 + 1e-6) apart, so the cells of a contact's centres differ by at most
// one. Coordinates beyond 2^27 cells and non-finite ones take the FP64 path.
static __device__ __noinline__ float2 bin_slow(double x, double H, double invH) {
  const int c = (int)floor(x * invH);
  return make_float2(__int_as_float(c), (float)(x - (double)c * H));
}
__device__ __forceinline__ void bin_axis(double x, double H, double invH, int &c, float &off) {
  constexpr uint32_t BIAS_HI = 0x41B80000u; // 1.5 * 2^28
  const double u = fma(x, invH, __hiloint2double((int)BIAS_HI, 0));
  const uint32_t hi = (uint32_t)__double2hiint(u), lo = (uint32_t)__double2loint(u);
  if ((hi >> 20) == (BIAS_HI >> 20)) {
    c = (int)__funnelshift_r(lo, hi - BIAS_HI, 24);
    off = (float)(lo & 0xFFFFFFu) * (1.0f / 16777216.0f) * (float)H;
    return;
  }
  const float2 s = bin_slow(x, H, invH);
  c = __float_as_int(s.x);
  off = s.y;
}

// The body's record and its entry in the hash grid; counters set for the
// step's search. x, y: the centre.
__device__ __forceinline__ void bin_body(const BinArgs &A, int64_t i, double x, double y) {
  const double ri = A.r[i];
  const float rf = narrow_trunc(ri), xf = narrow_trunc(x), yf = narrow_trunc(y);
  uint32_t flags = A.fixed[i] ? REL_FIXED : 0u;
  for (int k = 0; k < A.nplanes; ++k) {
    // n . (x - x_plane) <= r: decided in FP32 when the margin exceeds the
    // error of truncated coordinates and FP32 sums (under 1e-6 of the terms),
    // else in FP64 as the reference does
    const float ex = xf - A.pxf[k][0], ey = yf - A.pxf[k][1];
    const float gap = A.pnf[k][0] * ex + A.pnf[k][1] * ey - rf;
    const float err = 1.0e-6f * (fabsf(xf) + fabsf(A.pxf[k][0]) + fabsf(yf) +
                                 fabsf(A.pxf[k][1]) + rf);
    bool on;
    if (fabsf(gap) > err) {
      on = gap < 0.0f;
    } else {
      const double d = A.pn[k][0] * (x - A.px[k][0]) + A.pn[k][1] * (y - A.px[k][1]);
      on = d <= ri;
    }
    if (on) flags |= REL_PLANE0 << k;
  }
  // StaticDrumCircleConstraint::isActive (StaticDrumCircleConstraint.cpp:7-13):
  // |x_drum - x|^2 >= (r_drum - r)^2; drum k is static object nplanes + k
  for (int k = 0; k < A.ndrums; ++k) {
    const double ex = A.dx[k][0] - x, ey = A.dx[k][1] - y, g = A.dr[k] - ri;
    if (ex * ex + ey * ey >= g * g) flags |= REL_PLANE0 << (A.nplanes + k);
  }
  int cx, cy;
  float ox, oy;
  bin_axis(x, A.H, A.invH, cx, ox);
  bin_axis(y, A.H, A.invH, cy, oy);
  const int next = atomicExch(&A.heads[cell_bucket(cx, cy, A.mask)], (int)i);
  A.rec[2 * i] = make_float4(ox, oy, rf, __uint_as_float(flags));
  A.rec[2 * i + 1] =
      make_float4(__int_as_float(cx), __int_as_float(cy), __int_as_float(next), 0.0f);
  // fixed bodies have no contacts of their own
  const int ns = (flags & REL_FIXED) ? 0 : __popc(flags >> 1);
  A.pc[i] = (unsigned long long)ns;
  A.in_count[i] = 0;
  if (A.tiles && ns) atomicAdd(A.tiles + 4 * (i >> A.tile_shift), ns);
}

} // namespace hg
