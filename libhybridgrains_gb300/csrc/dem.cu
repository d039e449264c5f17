// Penalty-DEM disk step (PenaltyImpactFrictionMap::flow / flowWithWeights,
// rigidbody2d/PenaltyImpactFrictionMap.cpp:1083-1149) in FP64.
//
// Compiled with --fmad=false: every record and force is evaluated with the
// operation order of the reference's Eigen expressions, and body forces are
// summed in the reference's order (gravity, plane contacts, circle-circle
// contacts in (first, second) order, kinematic contacts) by a per-body gather
// instead of atomics. The step is therefore deterministic and matches a serial
// FP64 evaluation of the reference bit for bit.
//
// Kernels per step (in one of two ways to the tile sums):
//   kd_bin         broadphase: a hash grid of linked lists over the disks'
//                  centres, only in the first step after the bodies changed
//                  (later ones are binned by the integration). The cell width
//                  is 2 r_max (1 + 1e-6), so the partners of a disk lie in
//                  3x3 cells; the result is the reference's candidate set
//                  {i < j : AABBs overlap} (SpatialGrid.cpp:14-19, 90-118),
//                  independent of the reference's own cell width.
//   kd_pairs       narrow phase (RigidBody2DSim.cpp:270-336 with q0 == q1,
//                  CollisionDetectionUtilities.cpp:3-101) and body-plane
//                  tests (RigidBody2DSim.cpp:777-842): counts, keeping short
//                  partner lists. Candidates are filtered in FP32 on
//                  cell-relative offsets before the exact FP64 tests; the
//                  filter leaves about one FP64 test per contact at the
//                  filter's edge.
//   kd_pairs_emit  offsets and sorted per-body contact lists
//   kd_contacts    collision-cache update with tangential-spring carry
//                  (PenaltyImpactFrictionMap.cpp:296-599) and the penalty
//                  force with Coulomb projection (616-1081,
//                  secondRootOfQuadratic 601-614); incoming contact lists per
//                  body.
//   kd_integrate   force gather, fixed-body zeroing and symplectic Euler
//                  (PenaltyImpactFrictionMap.cpp:1101-1114), then the binning
//                  for the next step.
// Small scenes are bound by the chain of dependent launches and loads, the
// contact law by the FP64 pipe, a million disks by the records' 176 bytes per
// contact. Against a counting sort of the grid, scans for every offset list
// and records stored by their lanes (14 launches per step), per step: 1,000
// disks stepped one call at a time 63.6 -> 25.7 us; 10,000 disks at 2.8
// contacts each, FP64, 68.3 -> 28.5 us; 1,000,000 such disks, mixed, 889 ->
// 398 us.
#include "hg_internal.cuh"
#include "dem_bins.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

namespace hg {

namespace {

enum { K_PLANE = 0, K_CC = 1, K_KIN = 2 };
constexpr int RW = HG_DEM_RECORD_WIDTH;

struct D2 {
  double x, y;
};
__device__ __forceinline__ D2 dadd(D2 a, D2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ D2 dsub(D2 a, D2 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ D2 dscl(double s, D2 a) { return {s * a.x, s * a.y}; }
__device__ __forceinline__ double ddot(D2 a, D2 b) { return a.x * b.x + a.y * b.y; }
__device__ __forceinline__ double dsq(D2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double dnorm(D2 a) { return sqrt(dsq(a)); }
__device__ __forceinline__ D2 dnormalized(D2 a) {
  const double n2 = dsq(a);
  if (n2 > 0.0) {
    const double n = sqrt(n2);
    return {a.x / n, a.y / n};
  }
  return a;
}
__device__ __forceinline__ double dcross(D2 a, D2 b) { return a.x * b.y - a.y * b.x; }
__device__ __forceinline__ uint32_t cell_hash(int cx, int cy, uint32_t mask) {
  return ((uint32_t)cx * 73856093u ^ (uint32_t)cy * 19349663u) & mask;
}

__device__ __forceinline__ int64_t ckey(int kind, int a, int b) {
  return ((int64_t)kind << 60) | ((int64_t)a << 30) | (int64_t)b;
}

struct BroadArgs {
  int64_t n;
  double H; // cell width
  uint32_t mask;
  const double *mn; // 2 per box (min x, min y)
  const double *mx;
};

__global__ void kd_home(BroadArgs B, int2 *home, int32_t *bucket_count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= B.n) return;
  const int cx = (int)floor(B.mn[2 * i] / B.H), cy = (int)floor(B.mn[2 * i + 1] / B.H);
  home[i] = make_int2(cx, cy);
  atomicAdd(&bucket_count[cell_hash(cx, cy, B.mask)], 1);
}

__global__ void kd_fill(BroadArgs B, const int2 *__restrict__ home,
                        const int32_t *__restrict__ bucket_start, int32_t *cursor,
                        int32_t *items) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= B.n) return;
  const int2 c = home[i];
  const uint32_t b = cell_hash(c.x, c.y, B.mask);
  items[bucket_start[b] + atomicAdd(&cursor[b], 1)] = (int32_t)i;
}

// AABB::overlaps (SpatialGrid.cpp:14-19), inclusive on every side.
__device__ __forceinline__ bool box_overlap(const BroadArgs &B, int64_t i, int64_t j) {
  return (B.mx[2 * i] >= B.mn[2 * j] && B.mx[2 * i + 1] >= B.mn[2 * j + 1]) &&
         (B.mx[2 * j] >= B.mn[2 * i] && B.mx[2 * j + 1] >= B.mn[2 * i + 1]);
}

__device__ __forceinline__ void sort_small(int *keys, int n) {
  for (int i = 1; i < n; ++i) {
    const int k = keys[i];
    int j = i - 1;
    while (j >= 0 && keys[j] > k) {
      keys[j + 1] = keys[j];
      --j;
    }
    keys[j + 1] = k;
  }
}

// Bins every body: the first step after the bodies changed. Later steps find
// the bins made by the integration of the step before.
__global__ void __launch_bounds__(128) kd_bin(const __grid_constant__ BinArgs A,
                                              const double *q) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  bin_body(A, i, q[3 * i], q[3 * i + 1]);
}

// The per-body terms of kd_integrate that change only with the masses, the
// weights or the time step, with kd_integrate's operations: the gravity
// force 0 + M g (NearEarthGravityForce::computeForce) and dt / M, dt / Mi
// written as dt * (1 / M) (M = m0 w, Mi = I0 w:
// RigidBody2DState::updateCurrentMassUsingMassWeights).
__global__ void kd_body_terms(int64_t n, double dt, double gx, double gy,
                              const double *__restrict__ m0, const double *__restrict__ I0,
                              const double *__restrict__ w, double4 *terms) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double M = m0[j] * w[j], Mi = I0[j] * w[j];
  terms[j] = make_double4(0.0 + M * gx, 0.0 + M * gy, dt * (1.0 / M), dt * (1.0 / Mi));
}

constexpr int PW = 8; // partners per body kept by the search

struct PairArgs {
  int64_t n;
  uint32_t mask;
  const float4 *rec; // body records of bin_body
  float Hf;  // cell width in FP32
  float tol; // FP32 filter slack
  const int32_t *heads;
  const double *q;
  const double *r;
  int nstatic;            // static objects: the planes, then the drums
  unsigned long long *pc; // contact counts per first body
  int32_t *in_count;      // contacts per second body
  uint32_t *plist;        // PW partners per body (fixed partners flagged by bit 31)
  int4 *desc;   // per body: offsets of its static, circle-circle and kinematic
                // contacts and of its incoming list
  int32_t *descn; // per body: the three counts, 8 bits each
  int32_t *in_cursor;
  int32_t *tiles; // sums of the four counts over tiles of 2^tile_shift bodies
  int tile_shift, ntiles;
  bool add_tiles; // the search adds to tiles (else kd_tile_sums forms them)
  int64_t *keys; // contact keys, sorted
  int64_t ccap;
  int32_t *count; // total number of contacts
  int2 *range;    // [x, y): the circle-circle contacts
  uint32_t *status;
};

// The contact test of a candidate pair (a, b), b's home cell offset by
// (dx, dy) from a's. The FP32 offsets from the home cells' corners give the
// centre distance to within about 1e-6 of a cell (offsets and truncated radii
// to 1.2e-7 each, three FP32 sums); the slack tol is 4e-6 of a cell. So a pair
// whose FP32 distance exceeds ra + rb + tol is no contact, and one whose FP32
// distance is below ra + rb - tol is a contact under the reference's FP64
// tests as well (its AABBs overlap and c0 < 0 by about 2 tol (ra + rb), far
// beyond FP64 rounding). Only the pairs in between take those tests: AABB
// overlap (SpatialGrid.cpp:14-19, with the AABB corners x -+ r evaluated as
// CircleGeometry.cpp:22-30 does) and ballBallCCDCollisionHappens with q0 == q1
// (active iff c0 <= 0). A pair in between costs its warp a microsecond (a dozen
// FP64 instructions after four dependent loads), so the slack is small.
__device__ __forceinline__ bool is_contact(const PairArgs &A, float4 pa, float4 pb, int dx,
                                           int dy, int a, int b) {
  const float ex = (float)dx * A.Hf + (pb.x - pa.x);
  const float ey = (float)dy * A.Hf + (pb.y - pa.y);
  const float d2 = ex * ex + ey * ey;
  const float outer = pa.z + pb.z + A.tol, inner = pa.z + pb.z - A.tol;
  if (d2 > outer * outer) return false;
  if (inner > 0.0f && d2 < inner * inner) return true;
  const double xa = A.q[3 * a], ya = A.q[3 * a + 1], ra = A.r[a];
  const double xb = A.q[3 * b], yb = A.q[3 * b + 1], rb = A.r[b];
  if (!((xa + ra >= xb - rb && ya + ra >= yb - rb) && (xb + rb >= xa - ra && yb + rb >= ya - ra)))
    return false;
  const double ddx = xa - xb, ddy = ya - yb;
  const double c0 = (ddx * ddx + ddy * ddy) - (ra + rb) * (ra + rb);
  return c0 <= 0.0;
}

// Walks the bucket list from body b over the bodies whose home cell is (cx, cy)
// (a bucket may be shared by other cells).
template <class F>
__device__ __forceinline__ void for_each_in_cell(const PairArgs &A, int b, int cx, int cy,
                                                 F &&body) {
  // (a list holds each body once: the bound on the steps is never reached)
  for (int64_t left = A.n; b >= 0 && left > 0; --left) {
    if (!HG_INDEX_OK(b, A.n, A.status)) return;
    const float4 pb = A.rec[2 * b], cb = A.rec[2 * b + 1];
    if (__float_as_int(cb.x) == cx && __float_as_int(cb.y) == cy) body(b, pb);
    b = __float_as_int(cb.z);
  }
}

// Contact enumeration for body a as the first index: circle-circle with
// b > a non-fixed, kinematic with b fixed (any index; the reference swaps the
// fixed body into the second slot). Fixed bodies emit none. The 3x3 cells
// around a's home cell hold every candidate.
template <class F>
__device__ __forceinline__ void for_each_partner(const PairArgs &A, int a, F &&found) {
  const float4 pa = A.rec[2 * a], ca = A.rec[2 * a + 1];
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) {
      const int cx = __float_as_int(ca.x) + dx, cy = __float_as_int(ca.y) + dy;
      for_each_in_cell(A, A.heads[cell_bucket(cx, cy, A.mask)], cx, cy, [&](int b, float4 pb) {
        if (b == a) return;
        const bool bf = (__float_as_uint(pb.w) & REL_FIXED) != 0u;
        if (!(b > a || bf)) return;
        if (is_contact(A, pa, pb, dx, dy, a, b)) found(b, bf);
      });
    }
}

// Search over half of each neighbourhood: the home cell and the four cells
// after it in (dy, dx) order. A pair of bodies in different cells is met from
// exactly one of them (the offset from one home cell to the other is in the
// half, its negative is not); a pair within one cell is met from both and
// kept from the lower index. Each contact is credited to its first body (the
// lower index of two free bodies, the free body of a free-fixed pair, none
// for two fixed bodies): the count of its kind and the first PW partners in
// plist (in no particular order; the emission pass sorts them).
// Circle-circle contacts also count as incoming at their second body.

// Contacts found by a thread: kept until HELD of them can be credited together
// (an atomic's return is a round trip to L2: they overlap).
constexpr int HELD = 4;
struct Found {
  int first[HELD];
  uint32_t second[HELD]; // a kinematic (fixed) second flagged by bit 31
  int n;
  bool overflow;
};

// Adds one to tile t's count of kind comp for every calling lane with on set:
// one atomic per distinct count among the lanes of mask. (With one atomic per
// contact, 180 on each address at 10,000 disks, the search took 11.0 us instead
// of 8.0.)
__device__ __forceinline__ void add_tile(int32_t *tiles, unsigned mask, int t, int comp, bool on) {
  const int at = 4 * t + comp;
  const unsigned same = __match_any_sync(mask, at);
  const unsigned add = same & __ballot_sync(mask, on);
  const int lane = threadIdx.x & 31;
  if (add && lane == __ffs(same) - 1) atomicAdd(tiles + at, __popc(add));
}

__device__ __forceinline__ void credit(const PairArgs &A, Found &f) {
  unsigned long long p[HELD];
#pragma unroll
  for (int k = 0; k < HELD; ++k)
    if (k < f.n)
      p[k] = atomicAdd(A.pc + f.first[k], 1ull << (f.second[k] >> 31 ? PC_KIN : PC_CC));
#pragma unroll
  for (int k = 0; k < HELD; ++k) {
    if (k >= f.n) break;
    const int first = f.first[k], second = (int)(f.second[k] & 0x7FFFFFFFu);
    const bool kin = f.second[k] >> 31;
    const int ncc = pc_found_cc(p[k]), nkin = pc_found_kin(p[k]);
    const bool kept = (kin ? nkin : ncc) < MAXP;
    f.overflow |= !kept;
    if (ncc + nkin < PW) A.plist[(int64_t)first * PW + ncc + nkin] = f.second[k];
    if (!kin) atomicAdd(A.in_count + second, 1);
    if (A.add_tiles) {
      const unsigned mask = __activemask();
      add_tile(A.tiles, mask, first >> A.tile_shift, kin ? 2 : 1, kept);
      add_tile(A.tiles, mask, second >> A.tile_shift, 3, !kin);
    }
  }
  f.n = 0;
}

// cell c of the half neighbourhood: (0, 0), (1, 0), (-1, 1), (0, 1), (1, 1)
__device__ __forceinline__ int half_dx(int c) { return c == 0 ? 0 : (c == 1 ? 1 : c - 3); }
__device__ __forceinline__ int half_dy(int c) { return c >= 2 ? 1 : 0; }

__device__ __forceinline__ void search_cell(const PairArgs &A, int a, int c, float4 pa, int hx,
                                            int hy, int head, Found &f) {
  const bool af = (__float_as_uint(pa.w) & REL_FIXED) != 0u;
  const int dx = half_dx(c), dy = half_dy(c);
  for_each_in_cell(A, head, hx + dx, hy + dy, [&](int b, float4 pb) {
    if (b == a || (c == 0 && b < a)) return;
    const bool bf = (__float_as_uint(pb.w) & REL_FIXED) != 0u;
    if (af && bf) return;
    if (!is_contact(A, pa, pb, dx, dy, a, b)) return;
    const int first = af ? b : (bf ? a : min(a, b));
    const uint32_t second = af ? (uint32_t)a | 0x80000000u
                               : (bf ? (uint32_t)b | 0x80000000u : (uint32_t)max(a, b));
    if (!HG_INDEX_OK(first, A.n, A.status)) return;
    if (f.n == HELD) credit(A, f);
#pragma unroll
    for (int k = 0; k < HELD; ++k)
      if (k == f.n) {
        f.first[k] = first;
        f.second[k] = second;
      }
    ++f.n;
  });
}

// One thread per body over its five cells: fewer loads of the body's own
// record than kd_pairs when the bodies alone fill the GPU.
__global__ void __launch_bounds__(128) kd_pairs_body(const __grid_constant__ PairArgs A) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  const int a = (int)(blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
  if (a >= A.n) return;
  const float4 pa = A.rec[2 * a], ca = A.rec[2 * a + 1];
  const int hx = __float_as_int(ca.x), hy = __float_as_int(ca.y);
  Found f;
  f.n = 0;
  f.overflow = false;
  int head[5];
#pragma unroll
  for (int c = 0; c < 5; ++c)
    head[c] = A.heads[cell_bucket(hx + half_dx(c), hy + half_dy(c), A.mask)];
#pragma unroll
  for (int c = 0; c < 5; ++c) search_cell(A, a, c, pa, hx, hy, head[c], f);
  credit(A, f);
  if (f.overflow) atomicOr(A.status, (uint32_t)HG_STATUS_CELL_OVERFLOW);
}

// One thread per (body, cell of the half neighbourhood): thread t takes cell
// t / n of body t % n, so a warp's lanes read consecutive bodies' records and
// each thread follows one list instead of five.
__global__ void __launch_bounds__(128) kd_pairs(const __grid_constant__ PairArgs A) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  const int n = (int)A.n;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x); // 5 n < 2^31 here
  if (t >= 5 * n) return;
  const int c = t / n, a = t - c * n;
  const float4 pa = A.rec[2 * a], ca = A.rec[2 * a + 1];
  const int hx = __float_as_int(ca.x), hy = __float_as_int(ca.y);
  Found f;
  f.n = 0;
  f.overflow = false;
  search_cell(A, a, c, pa, hx, hy, A.heads[cell_bucket(hx + half_dx(c), hy + half_dy(c), A.mask)],
              f);
  credit(A, f);
  if (f.overflow) atomicOr(A.status, (uint32_t)HG_STATUS_CELL_OVERFLOW);
}

__device__ __forceinline__ int warp_sum(int x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
  return x;
}

// Sums of the contact counts (static, circle-circle, kinematic, incoming)
// over tiles of 2^shift bodies, one CTA per tile.
__global__ void __launch_bounds__(256) kd_tile_sums(int64_t n, int shift,
                                                    const unsigned long long *pc,
                                                    const int32_t *in_count,
                                                    int32_t *tiles) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  __shared__ int s_sum[8][4];
  const int64_t b0 = (int64_t)blockIdx.x << shift;
  const int64_t b1 = min(n, b0 + ((int64_t)1 << shift));
  int s[4] = {0, 0, 0, 0};
  for (int64_t i = b0 + threadIdx.x; i < b1; i += 256) {
    const unsigned long long p = pc[i];
    s[0] += pc_static(p);
    s[1] += pc_cc(p);
    s[2] += pc_kin(p);
    s[3] += in_count[i];
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int t = warp_sum(s[k]);
    if (lane == 0) s_sum[wid][k] = t;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    int t = 0;
    for (int w = 0; w < 8; ++w) t += s_sum[w][threadIdx.x];
    tiles[4 * (int64_t)blockIdx.x + threadIdx.x] = t;
  }
}

// Emission pass, one CTA per NT bodies: the offsets of their contacts, then
// their sorted contact keys. The offsets need no scan launches: a CTA sums
// the tile counts before its bodies itself (at most MAX_TILES of them), then
// the bodies between its tile's start and its first body, and scans its own.
// When the total exceeds the contact capacity the step keeps no contacts and
// reports HG_STATUS_CONTACT_OVERFLOW instead of writing past the buffers.
// Partner lists of at most PW bodies come from the search; longer ones are
// searched again (the same partners, the first MAXP of each kind).
constexpr int MAX_TILES = 1024;
template <int NT> __global__ void __launch_bounds__(NT) kd_pairs_emit(PairArgs A) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  constexpr int NW = NT / 32;
  __shared__ int s_sum[NW][7];
  __shared__ unsigned long long s_scan[NW];
  __shared__ int s_in[NW];
  const int64_t n = A.n;
  const int64_t b0 = blockIdx.x * (int64_t)NT;
  const int64_t a64 = b0 + threadIdx.x;
  const int a = (int)a64;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long p = a64 < n ? A.pc[a] : 0ull;
  const int nin = a64 < n ? A.in_count[a] : 0;
  // [0, 3): totals of the three kinds; [3, 7): counts before this CTA
  int sum[7] = {0, 0, 0, 0, 0, 0, 0};
  const int64_t t0 = b0 >> A.tile_shift;
  for (int t = threadIdx.x; t < A.ntiles; t += NT) {
    const int4 v = reinterpret_cast<const int4 *>(A.tiles)[t];
    const bool before = t < t0;
    sum[0] += v.x;
    sum[1] += v.y;
    sum[2] += v.z;
    sum[3] += before ? v.x : 0;
    sum[4] += before ? v.y : 0;
    sum[5] += before ? v.z : 0;
    sum[6] += before ? v.w : 0;
  }
  for (int64_t i = (t0 << A.tile_shift) + threadIdx.x; i < b0; i += NT) {
    const unsigned long long pi = A.pc[i];
    sum[3] += pc_static(pi);
    sum[4] += pc_cc(pi);
    sum[5] += pc_kin(pi);
    sum[6] += A.in_count[i];
  }
  // the CTA's own counts: three 21-bit fields scanned in one word
  const unsigned long long own = (unsigned long long)pc_static(p) |
                                 (unsigned long long)pc_cc(p) << 21 |
                                 (unsigned long long)pc_kin(p) << 42;
  unsigned long long inc = own;
  int inc_in = nin;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, inc, d);
    const int y = __shfl_up_sync(0xffffffffu, inc_in, d);
    if (lane >= d) {
      inc += x;
      inc_in += y;
    }
  }
  if (lane == 31) {
    s_scan[wid] = inc;
    s_in[wid] = inc_in;
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    const int t = warp_sum(sum[k]);
    if (lane == 0) s_sum[wid][k] = t;
  }
  __syncthreads();
  unsigned long long ex = inc - own;
  int ex_in = inc_in - nin;
#pragma unroll
  for (int k = 0; k < 7; ++k) sum[k] = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    if (w < wid) {
      ex += s_scan[w];
      ex_in += s_in[w];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) sum[k] += s_sum[w][k];
  }
  const bool over = (int64_t)sum[0] + sum[1] + sum[2] > A.ccap;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (over) atomicOr(A.status, (uint32_t)HG_STATUS_CONTACT_OVERFLOW);
    *A.count = over ? 0 : sum[0] + sum[1] + sum[2];
    *A.range = over ? make_int2(0, 0) : make_int2(sum[0], sum[0] + sum[1]);
  }
  if (a64 >= n) return;
  if (over) p = 0ull;
  const int npl = pc_static(p), ncc = pc_cc(p), nkin = pc_kin(p);
  const int64_t o0 = sum[3] + (int)(ex & 0x1FFFFFu);
  const int64_t o1 = (int64_t)sum[0] + sum[4] + (int)((ex >> 21) & 0x1FFFFFu);
  const int64_t o2 = (int64_t)sum[0] + sum[1] + sum[5] + (int)(ex >> 42);
  A.desc[a] = over ? make_int4(0, 0, 0, 0) : make_int4((int)o0, (int)o1, (int)o2, sum[6] + ex_in);
  A.descn[a] = npl | ncc << 8 | nkin << 16;
  A.in_cursor[a] = 0;
  if (npl + ncc + nkin == 0) return;
  if (o0 + npl > A.ccap || o1 + ncc > A.ccap || o2 + nkin > A.ccap) {
    atomicOr(A.status, (uint32_t)HG_STATUS_CONTACT_OVERFLOW);
    return;
  }
  const uint32_t flags = __float_as_uint(A.rec[2 * a].w);
  int j = 0;
  for (int k = 0; k < A.nstatic; ++k)
    if (flags & (REL_PLANE0 << k)) {
      if (j < npl) A.keys[o0 + j] = ckey(K_PLANE, a, k);
      ++j;
    }
  if (ncc + nkin <= PW) {
    // odd-even transposition sort of the flagged indices: circle-circle
    // partners ascending, then the fixed ones ascending
    uint32_t L[PW];
    const uint32_t *lst = A.plist + (int64_t)a * PW;
#pragma unroll
    for (int k = 0; k < PW; ++k) L[k] = k < ncc + nkin ? lst[k] : 0xFFFFFFFFu;
#pragma unroll
    for (int p = 0; p < PW; ++p)
#pragma unroll
      for (int i = p & 1; i + 1 < PW; i += 2) {
        const uint32_t lo = min(L[i], L[i + 1]), hi = max(L[i], L[i + 1]);
        L[i] = lo;
        L[i + 1] = hi;
      }
#pragma unroll
    for (int k = 0; k < PW; ++k) {
      if (k < ncc) A.keys[o1 + k] = ckey(K_CC, a, (int)L[k]);
      else if (k < ncc + nkin) A.keys[o2 + (k - ncc)] = ckey(K_KIN, a, (int)(L[k] & 0x7FFFFFFFu));
    }
    return;
  }
  int cc[MAXP], kin[MAXP];
  int mc = 0, mk = 0;
  for_each_partner(A, a, [&](int b, bool bf) {
    if (bf) {
      if (mk < MAXP) kin[mk++] = b;
    } else if (mc < MAXP) {
      cc[mc++] = b;
    }
  });
  sort_small(cc, mc);
  sort_small(kin, mk);
  for (int k = 0; k < min(mc, ncc); ++k) A.keys[o1 + k] = ckey(K_CC, a, cc[k]);
  for (int k = 0; k < min(mk, nkin); ++k) A.keys[o2 + k] = ckey(K_KIN, a, kin[k]);
}

struct ContactArgs {
  int64_t n;
  double dt;
  int weighted;
  double kn, kt, gn, gt, mu;
  double half_gn, half_gt;
  float mu2_32; // mu^2
  int nplanes;
  double px[HG_MAX_PLANES][2], pn[HG_MAX_PLANES][2];
  int ndrums; // static objects nplanes .. nplanes + ndrums - 1
  double dx[HG_MAX_DRUMS][2], dr[HG_MAX_DRUMS];
  const double *q, *v, *r, *w;
  const int32_t *count; // device count (total contacts)
  const int64_t *keys;
  double *rec;
  // per contact, for the integration: the total force and its torques about
  // the first and the second body (double4 in FP64, float4 in MIXED)
  void *load;
  const int4 *desc; // offsets of the bodies' contact lists (incoming: w)
  int32_t *in_cursor, *in_list;
  // the previous step's contacts; old_desc (with old_descn) gives each
  // body's lists in them, or is nullptr when the bodies were renumbered since
  const int64_t *old_keys;
  const double *old_rec;
  const int32_t *old_count;
  const int4 *old_desc;
  const int32_t *old_descn;
  // cleared for the next step: the search is done with them
  int32_t *heads, *tiles;
  int64_t nheads;
  int64_t ccap;
  uint32_t *status;
};

// The previous step's contact with this key: among its first body's own
// contacts of the kind (a few consecutive keys), or by binary search.
__device__ __forceinline__ int find_old(const ContactArgs &C, int64_t key, int kind, int a) {
  if (C.old_desc) {
    const int4 d = C.old_desc[a];
    const int n = (C.old_descn[a] >> (8 * kind)) & 0xFF;
    const int o = kind == K_PLANE ? d.x : (kind == K_CC ? d.y : d.z);
    for (int i = 0; i < n; ++i)
      if (C.old_keys[o + i] == key) return o + i;
    return -1;
  }
  int lo = 0, hi = min((int64_t)*C.old_count, C.ccap) - 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const int64_t k = C.old_keys[mid];
    if (k == key) return mid;
    if (k < key) lo = mid + 1;
    else hi = mid - 1;
  }
  return -1;
}

// secondRootOfQuadratic (PenaltyImpactFrictionMap.cpp:601-614)
__device__ __forceinline__ double second_root(double a, double b, double c, double ds) {
  if (b > 0.0) return (2.0 * c) / (-b - ds);
  return (-b + ds) / (2.0 * a);
}

constexpr int CONTACT_THREADS = 128;
constexpr int CONTACT_WARPS = CONTACT_THREADS / 32;
constexpr int RW2 = RW / 2; // a record in 16-byte pieces
static_assert(RW % 2 == 0, "records are moved in 16-byte pieces");

// The contact law's grid-stride loop, shared by the two precisions. Contacts
// go to the warps in chunks of 32, chunk c to CTA c mod gridDim, so that few
// contacts spread over all SMs (the law is bound by each SM's FP64 pipe).
// law(k, key, kind, a, b, out) computes contact k's record into out (the
// caller's shared-memory row). A record is 176 bytes: written by its lane it
// would be 22 stores of 8 bytes in 32 different sectors each, so the warp's
// records are staged in shared memory and written as contiguous 16-byte pieces.
template <class Law>
__device__ __forceinline__ void for_each_contact(const ContactArgs &C, Law &&law) {
  __shared__ __align__(16) double s_rec[CONTACT_WARPS][32 * RW];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t tid = blockIdx.x * (int64_t)CONTACT_THREADS + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * CONTACT_THREADS;
  for (int64_t i = tid; i < C.nheads / 4; i += nthreads)
    reinterpret_cast<int4 *>(C.heads)[i] = make_int4(-1, -1, -1, -1);
  for (int64_t i = tid; i < MAX_TILES; i += nthreads)
    reinterpret_cast<int4 *>(C.tiles)[i] = make_int4(0, 0, 0, 0);
  const int64_t total = min((int64_t)*C.count, C.ccap);
  double *out = s_rec[wid] + lane * RW;
  for (int64_t c = blockIdx.x + (int64_t)gridDim.x * wid; 32 * c < total;
       c += (int64_t)gridDim.x * CONTACT_WARPS) {
    const int64_t k = 32 * c + lane;
    if (k < total) {
      const int64_t key = C.keys[k];
      const int kind = (int)(key >> 60);
      const int a = (int)((key >> 30) & 0x3FFFFFFF);
      const int b = (int)(key & 0x3FFFFFFF);
      if (HG_INDEX_OK(a, C.n, C.status) &&
          HG_INDEX_OK(b, kind == K_PLANE ? (int64_t)(C.nplanes + C.ndrums) : C.n, C.status)) {
        // the second body's list of incoming contacts (the slot arrives while
        // the law runs)
        int slot = 0, list = 0;
        if (kind == K_CC) {
          slot = atomicAdd(&C.in_cursor[b], 1);
          list = C.desc[b].w;
        }
        law(k, key, kind, a, b, out);
        if (kind == K_CC && (int64_t)list + slot < C.ccap) C.in_list[list + slot] = (int32_t)k;
      }
    }
    __syncwarp();
    const int pieces = (int)min((int64_t)32, total - 32 * c) * RW2;
    const double2 *src = reinterpret_cast<const double2 *>(s_rec[wid]);
    double2 *dst = reinterpret_cast<double2 *>(C.rec + 32 * c * RW);
    for (int i = lane; i < pieces; i += 32) dst[i] = src[i];
    __syncwarp();
  }
}

__device__ __forceinline__ void put2(double *out, int i, double x, double y) {
  reinterpret_cast<double2 *>(out)[i] = make_double2(x, y);
}

// FP32 estimate of |a|^2 from truncated components (0 for those below FP32's
// range); top: the largest exponent word met.
__device__ __forceinline__ float square_est(D2 a, uint32_t &top) {
  auto est = [&](double x) {
    const uint32_t hi = f64_hi(x) & 0x7FFFFFFFu;
    top = max(top, hi);
    const uint32_t f = __funnelshift_l(f64_lo(x), hi, 3) - (896u << 23);
    return __uint_as_float(hi < 897u << 20 ? 0u : f);
  };
  const float x = est(a.x), y = est(a.y);
  return x * x + y * y;
}

__global__ void __launch_bounds__(CONTACT_THREADS) kd_contacts(const __grid_constant__ ContactArgs C) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  for_each_contact(C, [&](int64_t k, int64_t key, int kind, int a, int b, double *out) {
    const D2 qa{C.q[3 * a], C.q[3 * a + 1]};
    const D2 va{C.v[3 * a], C.v[3 * a + 1]};
    const double wa = C.v[3 * a + 2];
    double depth, weight;
    D2 n, cp{0.0, 0.0}, r0, r1{0.0, 0.0}, vrel;
    const double ra = C.r[a];
    const int o = find_old(C, key, kind, a); // (its loads overlap the bodies')
    if (kind == K_PLANE && b >= C.nplanes) { // PenaltyImpactFrictionMap.cpp:361-401
      // StaticDrumCircleConstraint.cpp:100-159: the normal points from the
      // disk's centre to the drum's; the contact point is the disk's point
      // farthest from the drum's centre
      const int dk = b - C.nplanes;
      const D2 xd{C.dx[dk][0], C.dx[dk][1]};
      n = dnormalized(dsub(xd, qa));
      cp = dsub(qa, dscl(ra, n));
      weight = C.weighted ? C.w[a] : 1.0;
      const double gap = -(dnorm(dsub(xd, qa)) - (C.dr[dk] - ra));
      depth = gap < 0.0 ? gap : 0.0; // std::min(0.0, gap)
      r0 = dscl(-ra, n);
      const D2 t0{-r0.y, r0.x};
      const D2 arm = dsub(cp, xd);
      const D2 tp{-arm.y, arm.x};
      const D2 vp{0.0 + 0.0 * tp.x, 0.0 + 0.0 * tp.y}; // the drum is static
      vrel = dsub(dadd(va, dscl(wa, t0)), vp);
    } else if (kind == K_PLANE) { // PenaltyImpactFrictionMap.cpp:316-359
      const D2 xp{C.px[b][0], C.px[b][1]};
      n = D2{C.pn[b][0], C.pn[b][1]};
      cp = dsub(qa, dscl(ra, n));
      weight = C.weighted ? C.w[a] : 1.0;
      depth = min_zero(ddot(n, dsub(qa, xp)) - ra);
      r0 = dscl(-ra, n);
      const D2 t0{-r0.y, r0.x};
      const D2 arm = dsub(cp, xp);
      const D2 tp{-arm.y, arm.x};
      const D2 vp{0.0 + 0.0 * tp.x, 0.0 + 0.0 * tp.y};
      vrel = dsub(dadd(va, dscl(wa, t0)), vp);
    } else {
      const D2 qb{C.q[3 * b], C.q[3 * b + 1]};
      const double rb = C.r[b];
      const D2 d = dsub(qa, qb);
      const double d2 = dsq(d), dist = sqrt(d2);
      n = d;
      if (!f64_zero(d2)) {
        const Divisor len = divisor(dist);
        bool ok = len.ok;
        n = D2{quot(d.x, len, ok), quot(d.y, len, ok)};
        if (!ok) n = D2{divide(d.x, dist), divide(d.y, dist)};
      }
      depth = min_zero(dist - ra - rb);
      const D2 vb{C.v[3 * b], C.v[3 * b + 1]};
      const double wb = C.v[3 * b + 2];
      if (kind == K_CC) { // CircleCircleConstraint.cpp:171-233
        cp = dadd(qa, dscl(ra / (ra + rb), D2{-d.x, -d.y}));
        weight = C.weighted ? (C.w[a] + C.w[b]) * 0.5 : 1.0;
        r0 = dsub(cp, qa);
        r1 = dsub(cp, qb);
        const D2 t0{-r0.y, r0.x}, t1{-r1.y, r1.x};
        vrel = dsub(dsub(dadd(va, dscl(wa, t0)), vb), dscl(wb, t1));
      } else { // KinematicObjectCircleConstraint.cpp
        cp = dsub(qa, dscl(ra, n));
        weight = C.weighted ? C.w[a] : 1.0;
        r0 = dscl(-ra, n);
        const D2 t{-r0.y, r0.x};
        const D2 arm = dsub(cp, qb);
        const D2 tk{-arm.y, arm.x};
        const D2 vk = dadd(vb, dscl(wb, tk));
        vrel = dsub(dadd(va, dscl(wa, t)), vk);
      }
    }
    // tangential spring carry
    D2 ds;
    if (o >= 0) {
      const double2 old = *reinterpret_cast<const double2 *>(C.old_rec + (int64_t)o * RW + 6);
      ds = dadd(D2{old.x, old.y}, dscl(C.dt, vrel));
    } else {
      ds = dscl(C.dt, vrel);
    }
    ds = dsub(ds, dscl(ddot(n, ds), n));
    // penalty force (PenaltyImpactFrictionMap.cpp:616-1081)
    const double w = weight;
    // (products with a weight of 1 are the products without it)
    double nkn = -C.kn, nkt = -C.kt, hgn = C.half_gn, hgt = C.half_gt;
    if (__double_as_longlong(w) != __double_as_longlong(1.0)) {
      nkn = nkn * w;
      nkt = nkt * w;
      hgn = hgn * w;
      hgt = hgt * w;
    }
    const D2 vt = dsub(vrel, dscl(ddot(n, vrel), n));
    const D2 vn = dsub(vrel, vt);
    const D2 fn = dsub(dscl(nkn * depth, n), dscl(hgn, vn));
    D2 ft = dsub(dscl(nkt, ds), dscl(hgt, vt));
    // Coulomb's law compares gamma_t w / 2 |vt| and |ft| with mu |fn|. FP32
    // estimates of their squares, within 1e-6 of them, decide all but close
    // calls (2e-5): a sticking contact then needs none of the three square
    // roots, a sliding one none but the root of its quadratic.
    uint32_t top = 0u;
    const float vt2 = square_est(vt, top), fn2 = square_est(fn, top), ft2 = square_est(ft, top);
    const float half_gt32 = narrow_trunc(hgt);
    const float cap2 = C.mu2_32 * fn2, drag2 = half_gt32 * half_gt32 * vt2;
    const float low = fminf(fminf(vt2, fn2), fminf(ft2, cap2));
    const bool sure = top < 1063u << 20 && low > 1.0e-24f; // squares within FP32
    const bool stick_drag = sure && drag2 < cap2 * 0.99998f; // not slipping
    if (!(stick_drag && ft2 < cap2 * 0.99998f)) {
      bool slip = false, slide = true;
      double mu_fn = 0.0;
      if (!(stick_drag && ft2 > cap2 * 1.00002f)) {
        mu_fn = C.mu * dnorm(fn);
        slip = hgt * dnorm(vt) > mu_fn;
        slide = dnorm(ft) > mu_fn;
      }
      if (slip) {
        ds = D2{0.0, 0.0};
        ft = dscl(-0.5 * C.gt * w, vt);
        ft = dnormalized(ft);
        ft = dscl(mu_fn, ft);
      } else if (slide) {
        const double qa_ = C.kt * w * C.kt * w * dsq(ds);
        const double qb_ = C.kt * w * C.gt * w * ddot(ds, vt);
        const double qc_ = 0.25 * C.gt * w * C.gt * w * ddot(vt, vt) - C.mu * C.mu * dsq(fn);
        const double dscr = qb_ * qb_ - 4 * qa_ * qc_;
        const double root1 = second_root(qa_, qb_, qc_, sqrt(dscr));
        const D2 nds = dscl(root1, ds);
        ft = dsub(dscl(-C.kt * w, nds), dscl(0.5 * C.gt * w, vt));
        ds = nds;
      }
    }
    const D2 f = dadd(fn, ft);
    reinterpret_cast<double4 *>(C.load)[k] =
        make_double4(f.x, f.y, dcross(r0, f), kind == K_CC ? dcross(r1, f) : 0.0);
    put2(out, 0, index_f64(kind), index_f64(a));
    put2(out, 1, index_f64(b), depth);
    put2(out, 2, n.x, n.y);
    put2(out, 3, ds.x, ds.y);
    put2(out, 4, vrel.x, vrel.y);
    put2(out, 5, r0.x, r0.y);
    put2(out, 6, r1.x, r1.y);
    put2(out, 7, weight, cp.x);
    put2(out, 8, cp.y, fn.x);
    put2(out, 9, fn.y, ft.x);
    put2(out, 10, ft.y, 0.0);
  });
}

struct IntegrateArgs {
  int64_t n, ccap;
  double dt;
  double *q, *v;
  double *q_before; // receives the positions before the step, or nullptr
  const double4 *terms;
  const uint8_t *fixed;
  const int4 *desc;
  const int32_t *descn, *in_cursor;
  int32_t *in_list;
  const void *load;
  const int64_t *keys; // the contacts, and the circle-circle ones' range
  const int2 *range;
  uint32_t *status;
};

// Body j's contacts in the reference's order: with static objects, as the
// second body of circle-circle contacts (their first indices lie below j, so
// they come before j's own list in the reference's loop), as the first body,
// and with fixed disks. apply(load, as_second). The incoming list, filled in
// no particular order, is sorted first. The first four incoming and own loads
// are fetched together: the sums are a chain, their loads need not be.
// The lists have room for every contact found, so with more than MAXP on a body
// they can go past the buffer, which holds the contacts kept; such a body's are
// looked up among all circle-circle contacts (by second body, in order).
template <class L, class F>
__device__ __forceinline__ void for_each_load(const IntegrateArgs &A, int64_t j, F &&apply) {
  const L *load = reinterpret_cast<const L *>(A.load);
  const int4 d = A.desc[j];
  const int counts = A.descn[j];
  int nin = A.in_cursor[j];
  const int64_t ccap = A.ccap;
  uint32_t *status = A.status;
  const int ns = counts & 0xFF, ncc = (counts >> 8) & 0xFF, nkin = (counts >> 16) & 0xFF;
  const bool listed = (int64_t)d.w + nin <= ccap;
  int32_t *lst = A.in_list + d.w;
  int in[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) in[k] = k < nin && listed ? lst[k] : 0x7FFFFFFF;
  L own[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < ncc) own[k] = load[d.y + k];
  for (int k = 0; k < ns; ++k) apply(load[d.x + k], false);
  if (!listed) {
    const int2 r = *A.range;
    for (int64_t k = r.x; k < r.y && nin > 0; ++k)
      if ((int64_t)(A.keys[k] & 0x3FFFFFFF) == j) {
        apply(load[k], true);
        --nin;
      }
  } else if (nin <= 4) {
    auto order = [&](int x, int y) {
      const int lo = min(in[x], in[y]), hi = max(in[x], in[y]);
      in[x] = lo;
      in[y] = hi;
    };
    order(0, 1);
    order(2, 3);
    order(0, 2);
    order(1, 3);
    order(1, 2);
    L got[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nin && HG_INDEX_OK(in[k], ccap, status)) got[k] = load[in[k]];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nin && HG_INDEX_OK(in[k], ccap, status)) apply(got[k], true);
  } else {
    for (int i = 1; i < nin; ++i) {
      const int key = lst[i];
      int t = i - 1;
      while (t >= 0 && lst[t] > key) {
        lst[t + 1] = lst[t];
        --t;
      }
      lst[t + 1] = key;
    }
    for (int i = 0; i < nin; ++i)
      if (HG_INDEX_OK(lst[i], ccap, status)) apply(load[lst[i]], true);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < ncc) apply(own[k], false);
  for (int k = 4; k < ncc; ++k) apply(load[d.y + k], false);
  for (int k = 0; k < nkin; ++k) apply(load[d.z + k], false);
}

// Force gather and symplectic Euler. With BIN the body is binned at its new
// position for the next step's search (the tables were cleared by the contact
// law), which saves that step a pass over the bodies.
template <bool BIN>
__global__ void kd_integrate(const __grid_constant__ IntegrateArgs A,
                             const __grid_constant__ BinArgs B) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= A.n) return;
  // gravity and dt / M, dt / Mi from kd_body_terms
  const double4 bt = A.terms[j];
  const double u0 = A.v[3 * j], u1 = A.v[3 * j + 1], u2 = A.v[3 * j + 2];
  const double p0 = A.q[3 * j], p1 = A.q[3 * j + 1], p2 = A.q[3 * j + 2];
  const bool fixed = A.fixed[j] != 0;
  double Fx = bt.x, Fy = bt.y, T = 0.0;
  for_each_load<double4>(A, j, [&](const double4 &f, bool second) {
    if (second) {
      Fx -= f.x;
      Fy -= f.y;
      T -= f.w;
    } else {
      Fx += f.x;
      Fy += f.y;
      T += f.z;
    }
  });
  if (fixed) Fx = Fy = T = 0.0;
  // v1 = v0 + dt Minv F ; q1 = q0 + dt v1
  const double v0 = u0 + bt.z * Fx;
  const double v1 = u1 + bt.z * Fy;
  const double v2 = u2 + bt.w * T;
  A.v[3 * j] = v0;
  A.v[3 * j + 1] = v1;
  A.v[3 * j + 2] = v2;
  if (A.q_before) {
    A.q_before[3 * j] = p0;
    A.q_before[3 * j + 1] = p1;
    A.q_before[3 * j + 2] = p2;
  }
  const double q0 = p0 + A.dt * v0, q1 = p1 + A.dt * v1, q2 = p2 + A.dt * v2;
  A.q[3 * j] = q0;
  A.q[3 * j + 1] = q1;
  A.q[3 * j + 2] = q2;
  if (!finite_bits(q0) || !finite_bits(q1) || !finite_bits(v0) || !finite_bits(v1))
    atomicOr(A.status, (uint32_t)HG_STATUS_NONFINITE);
  if (BIN) bin_body(B, j, q0, q1);
}

// ---- mixed precision: the same contact law and integration with FP32
// arithmetic; positions, the pairwise position difference, the contact point
// and the position update stay FP64 (a millimetre overlap taken from
// metre-scale coordinates in FP32 would be lost to cancellation). Records and
// velocities keep the FP64 storage of the FP64 path, holding FP32 values, so
// the broadphase, history relabelling, collision-cache export, coupling and
// checkpoints are shared.
struct F2 {
  float x, y;
};
__device__ __forceinline__ F2 fadd(F2 a, F2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ F2 fsub(F2 a, F2 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ F2 fscl(float s, F2 a) { return {s * a.x, s * a.y}; }
__device__ __forceinline__ float fdot(F2 a, F2 b) { return a.x * b.x + a.y * b.y; }
__device__ __forceinline__ float fnrm(F2 a) { return sqrtf(fdot(a, a)); }
__device__ __forceinline__ F2 fnormalized(F2 a) {
  const float n2 = fdot(a, a);
  if (n2 > 0.0f) {
    const float n = sqrtf(n2);
    return {a.x / n, a.y / n};
  }
  return a;
}
__device__ __forceinline__ float fcross(F2 a, F2 b) { return a.x * b.y - a.y * b.x; }

__global__ void __launch_bounds__(CONTACT_THREADS) kdx_contacts(const __grid_constant__ ContactArgs C) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  const float dt = (float)C.dt, kn = (float)C.kn, kt = (float)C.kt, gn = (float)C.gn,
              gt = (float)C.gt, mu = (float)C.mu;
  for_each_contact(C, [&](int64_t k, int64_t key, int kind, int a, int b, double *out) {
    const double qax = C.q[3 * a], qay = C.q[3 * a + 1];
    const F2 va{narrow(C.v[3 * a]), narrow(C.v[3 * a + 1])};
    const float wa = narrow(C.v[3 * a + 2]);
    const float ra = narrow(C.r[a]);
    const int o = find_old(C, key, kind, a); // (its loads overlap the bodies')
    float depth, weight;
    F2 n, r0, r1{0.0f, 0.0f}, vrel;
    double cpx, cpy;
    if (kind == K_PLANE && b >= C.nplanes) { // PenaltyImpactFrictionMap.cpp:361-401
      const int dk = b - C.nplanes;
      const double ex = C.dx[dk][0] - qax, ey = C.dx[dk][1] - qay; // FP64 difference
      const F2 e{narrow(ex), narrow(ey)};
      n = fnormalized(e); // towards the drum's centre
      // -(|e| - (R - r)) as ((R - r)^2 - |e|^2) / (|e| + R - r): the
      // cancelling difference in FP64, the rest in FP32
      const double g = C.dr[dk] - C.r[a];
      const double g2 = g * g - (ex * ex + ey * ey);
      depth = g2 < 0.0 ? narrow(g2) / (fnrm(e) + narrow(g)) : 0.0f;
      weight = C.weighted ? narrow(C.w[a]) : 1.0f;
      r0 = fscl(-ra, n);
      cpx = qax + widen_f32(r0.x);
      cpy = qay + widen_f32(r0.y);
      vrel = fadd(va, fscl(wa, F2{-r0.y, r0.x})); // the drum is static
    } else if (kind == K_PLANE) { // PenaltyImpactFrictionMap.cpp:316-359
      n = F2{narrow(C.pn[b][0]), narrow(C.pn[b][1])};
      // penetration from FP64 positions (a difference of nearly equal terms)
      const double dist = C.pn[b][0] * (qax - C.px[b][0]) + C.pn[b][1] * (qay - C.px[b][1]);
      depth = narrow(min_zero(dist - C.r[a]));
      weight = C.weighted ? narrow(C.w[a]) : 1.0f;
      r0 = fscl(-ra, n);
      cpx = qax + widen_f32(r0.x);
      cpy = qay + widen_f32(r0.y);
      vrel = fadd(va, fscl(wa, F2{-r0.y, r0.x})); // the plane is static
    } else {
      const double qbx = C.q[3 * b], qby = C.q[3 * b + 1];
      const float rb = narrow(C.r[b]);
      const double dx = qax - qbx, dy = qay - qby; // FP64 difference
      const F2 d{narrow(dx), narrow(dy)};
      n = fnormalized(d);
      // |d| - (ra + rb) as (|d|^2 - (ra + rb)^2) / (|d| + ra + rb): the
      // cancelling difference in FP64, the rest in FP32
      const double rs = C.r[a] + C.r[b];
      const double g2 = (dx * dx + dy * dy) - rs * rs;
      depth = g2 < 0.0 ? narrow(g2) / (fnrm(d) + narrow(rs)) : 0.0f;
      const F2 vb{narrow(C.v[3 * b]), narrow(C.v[3 * b + 1])};
      const float wb = narrow(C.v[3 * b + 2]);
      if (kind == K_CC) { // CircleCircleConstraint.cpp:171-233
        weight = C.weighted ? narrow((C.w[a] + C.w[b]) * 0.5) : 1.0f;
        r0 = fscl(-(ra / (ra + rb)), d); // p - xa = ra/(ra+rb) (xb - xa)
        r1 = fadd(d, r0);                // p - xb
        vrel = fsub(fsub(fadd(va, fscl(wa, F2{-r0.y, r0.x})), vb), fscl(wb, F2{-r1.y, r1.x}));
      } else { // KinematicObjectCircleConstraint.cpp
        weight = C.weighted ? narrow(C.w[a]) : 1.0f;
        r0 = fscl(-ra, n);
        const F2 arm = fadd(d, r0); // p - xb
        const F2 vk = fadd(vb, fscl(wb, F2{-arm.y, arm.x}));
        vrel = fsub(fadd(va, fscl(wa, F2{-r0.y, r0.x})), vk);
      }
      cpx = qax + widen_f32(r0.x);
      cpy = qay + widen_f32(r0.y);
    }
    // tangential spring carry
    F2 ds;
    if (o >= 0) {
      const double2 old = *reinterpret_cast<const double2 *>(C.old_rec + (int64_t)o * RW + 6);
      ds = fadd(F2{narrow(old.x), narrow(old.y)}, fscl(dt, vrel));
    } else {
      ds = fscl(dt, vrel);
    }
    ds = fsub(ds, fscl(fdot(n, ds), n));
    // penalty force (PenaltyImpactFrictionMap.cpp:616-1081)
    const float w = weight;
    const F2 vt = fsub(vrel, fscl(fdot(n, vrel), n));
    const F2 vn = fsub(vrel, vt);
    const F2 fn = fsub(fscl(-kn * w * depth, n), fscl(0.5f * gn * w, vn));
    F2 ft = fsub(fscl(-kt * w, ds), fscl(0.5f * gt * w, vt));
    const float mu_fn = mu * fnrm(fn);
    if (0.5f * gt * w * fnrm(vt) > mu_fn) {
      ds = F2{0.0f, 0.0f};
      ft = fscl(mu_fn, fnormalized(fscl(-0.5f * gt * w, vt)));
    } else if (fnrm(ft) > mu_fn) {
      // secondRootOfQuadratic (PenaltyImpactFrictionMap.cpp:601-614)
      const float qa_ = kt * w * kt * w * fdot(ds, ds);
      const float qb_ = kt * w * gt * w * fdot(ds, vt);
      const float qc_ = 0.25f * gt * w * gt * w * fdot(vt, vt) - mu * mu * fdot(fn, fn);
      const float sq = sqrtf(fmaxf(qb_ * qb_ - 4.0f * qa_ * qc_, 0.0f));
      const float root1 = qb_ > 0.0f ? (2.0f * qc_) / (-qb_ - sq) : (-qb_ + sq) / (2.0f * qa_);
      ds = fscl(root1, ds);
      ft = fsub(fscl(-kt * w, ds), fscl(0.5f * gt * w, vt));
    }
    const F2 f = fadd(fn, ft);
    reinterpret_cast<float4 *>(C.load)[k] = make_float4(f.x, f.y, fcross(r0, f), fcross(r1, f));
    put2(out, 0, index_f64(kind), index_f64(a));
    put2(out, 1, index_f64(b), widen_f32(depth));
    put2(out, 2, widen_f32(n.x), widen_f32(n.y));
    put2(out, 3, widen_f32(ds.x), widen_f32(ds.y));
    put2(out, 4, widen_f32(vrel.x), widen_f32(vrel.y));
    put2(out, 5, widen_f32(r0.x), widen_f32(r0.y));
    put2(out, 6, widen_f32(r1.x), widen_f32(r1.y));
    put2(out, 7, widen_f32(weight), cpx);
    put2(out, 8, cpy, widen_f32(fn.x));
    put2(out, 9, widen_f32(fn.y), widen_f32(ft.x));
    put2(out, 10, widen_f32(ft.y), 0.0);
  });
}

// Force gather (the FP64 kernel's summation order) and symplectic Euler in
// FP32; q += dt v in FP64.
template <bool BIN>
__global__ void kdx_integrate(const __grid_constant__ IntegrateArgs A,
                              const __grid_constant__ BinArgs B) {
  // (launched with programmatic dependence on the kernel before it)
  pdl_wait();
  pdl_trigger();
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= A.n) return;
  const double4 bt = A.terms[j];
  const double u0 = A.v[3 * j], u1 = A.v[3 * j + 1], u2 = A.v[3 * j + 2];
  const double p0 = A.q[3 * j], p1 = A.q[3 * j + 1], p2 = A.q[3 * j + 2];
  const bool fixed = A.fixed[j] != 0;
  float Fx = narrow(bt.x), Fy = narrow(bt.y), T = 0.0f;
  for_each_load<float4>(A, j, [&](const float4 &f, bool second) {
    Fx += second ? -f.x : f.x;
    Fy += second ? -f.y : f.y;
    T += second ? -f.w : f.z;
  });
  if (fixed) Fx = Fy = T = 0.0f;
  const float v0 = narrow(u0) + narrow(bt.z) * Fx;
  const float v1 = narrow(u1) + narrow(bt.z) * Fy;
  const float v2 = narrow(u2) + narrow(bt.w) * T;
  const double w0 = widen_f32(v0), w1 = widen_f32(v1), w2 = widen_f32(v2);
  A.v[3 * j] = w0;
  A.v[3 * j + 1] = w1;
  A.v[3 * j + 2] = w2;
  if (A.q_before) {
    A.q_before[3 * j] = p0;
    A.q_before[3 * j + 1] = p1;
    A.q_before[3 * j + 2] = p2;
  }
  const double q0 = p0 + A.dt * w0, q1 = p1 + A.dt * w1, q2 = p2 + A.dt * w2;
  A.q[3 * j] = q0;
  A.q[3 * j + 1] = q1;
  A.q[3 * j + 2] = q2;
  if (!finite_bits(q0) || !finite_bits(q1) || !isfinite(v0) || !isfinite(v1))
    atomicOr(A.status, (uint32_t)HG_STATUS_NONFINITE);
  if (BIN) bin_body(B, j, q0, q1);
}


// Candidate pairs of explicit boxes (SpatialGrid::getPotentialOverlaps).
template <bool EMIT>
__global__ void kd_box_pairs(BroadArgs B, const int2 *__restrict__ home,
                             const int32_t *__restrict__ bstart,
                             const int32_t *__restrict__ bcount,
                             const int32_t *__restrict__ items, int32_t *cnt,
                             const int32_t *__restrict__ off, int32_t *pairs, int64_t cap,
                             uint32_t *status) {
  const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (a >= B.n) return;
  int list[MAXP];
  int np = 0;
  bool overflow = false;
  const int cx0 = (int)floor(B.mn[2 * a] / B.H) - 1, cy0 = (int)floor(B.mn[2 * a + 1] / B.H) - 1;
  const int cx1 = (int)floor(B.mx[2 * a] / B.H), cy1 = (int)floor(B.mx[2 * a + 1] / B.H);
  for (int cy = cy0; cy <= cy1; ++cy)
    for (int cx = cx0; cx <= cx1; ++cx) {
      const uint32_t bk = cell_hash(cx, cy, B.mask);
      for (int k = bstart[bk], e = bstart[bk] + bcount[bk]; k < e; ++k) {
        const int b = items[k];
        if (b <= a) continue;
        const int2 hb = home[b];
        if (hb.x != cx || hb.y != cy) continue;
        if (!box_overlap(B, a, b)) continue;
        if (np < MAXP) list[np++] = b;
        else overflow = true;
      }
    }
  if (overflow) atomicOr(status, (uint32_t)HG_STATUS_CELL_OVERFLOW);
  if (!EMIT) {
    cnt[a] = np;
    return;
  }
  sort_small(list, np);
  const int64_t o = off[a];
  for (int k = 0; k < np; ++k)
    if (o + k < cap) {
      pairs[2 * (o + k)] = (int32_t)a;
      pairs[2 * (o + k) + 1] = list[k];
    }
}

inline int blocks_for(int64_t n, int t) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }


// Hash table sizes: at least two buckets per box or body, and 16
uint32_t table_bits(int64_t n) {
  uint32_t bits = 4;
  while (((int64_t)1 << bits) < 2 * n && bits < 30) ++bits;
  return bits;
}

// Broadphase tables for n boxes: bucket counts/starts, items and home cells.
hg_status build_buckets(cudaStream_t s, BroadArgs &B, int32_t *bcount, int32_t *bstart,
                        int32_t *cursor, int32_t *items, int2 *home, int32_t *scan_tmp) {
  const int64_t T = (int64_t)B.mask + 1;
  HG_CUDA_TRY(cudaMemsetAsync(bcount, 0, sizeof(int32_t) * T, s));
  HG_CUDA_TRY(cudaMemsetAsync(cursor, 0, sizeof(int32_t) * T, s));
  if (B.n == 0) return HG_OK;
  HG_LAUNCH(kd_home, blocks_for(B.n, 256), 256, 0, s, B, home, bcount);
  HG_CHECK_LAUNCH();
  hg_status st = exclusive_scan_i32(bcount, bstart, T, scan_tmp, s);
  if (st != HG_OK) return st;
  HG_LAUNCH(kd_fill, blocks_for(B.n, 256), 256, 0, s, B, home, bstart, cursor, items);
  HG_CHECK_LAUNCH();
  return HG_OK;
}


} // namespace

namespace {

// tiles of at least 64 bodies, at most MAX_TILES of them
int tile_shift_for(int64_t n) {
  int sh = 6;
  while (((n - 1) >> sh) + 1 > MAX_TILES) ++sh;
  return sh;
}

} // namespace

// Below about one body per thread slot of the GPU, five threads per body
// hide the buckets' latency, and the search adds to the tile sums as it
// goes (a launch less); above it, one thread per body reads each body's
// record once, and the sums take a pass of their own (at a million disks
// under contact load the added atomics cost more than the pass).
static bool search_by_cells(const hg_dem *d) { return d->n < (int64_t)d->ctx->num_sms * 1024; }

hg_status dem_alloc(hg_dem *d) {
  const int64_t N = std::max<int64_t>(d->cap, 1);
  const int64_t C = std::max<int64_t>(d->ccap, 1);
  d->mask = (1u << table_bits(N)) - 1u;
  const int64_t T = (int64_t)d->mask + 1;
  const bool mixed = d->p.precision == HG_PRECISION_MIXED;
  hg_status st;
  if ((st = d->status.alloc(1)) || (st = d->q.alloc(3 * N)) || (st = d->v.alloc(3 * N)) ||
      (st = d->r.alloc(N)) || (st = d->m0.alloc(N)) || (st = d->I0.alloc(N)) ||
      (st = d->w.alloc(N)) || (st = d->minv.alloc(4 * N)) || (st = d->fixed.alloc(N)) ||
      (st = d->brec.alloc(2 * N)) || (st = d->plist.alloc(PW * N)) || (st = d->heads.alloc(T)) ||
      (st = d->pc.alloc(N)) || (st = d->in_count.alloc(N)) ||
      (st = d->tiles.alloc(4 * (int64_t)MAX_TILES)) || (st = d->c_count.alloc(2)) ||
      (st = d->cc_range.alloc(1)) || (st = d->in_list.alloc(C)) || (st = d->in_cursor.alloc(N)) ||
      (st = d->load.alloc(C * (mixed ? 16 : 32))))
    return st;
  for (int b = 0; b < 2; ++b)
    if ((st = d->ckey[b].alloc(C)) || (st = d->crec[b].alloc(C * RW)) ||
        (st = d->desc[b].alloc(N)) || (st = d->descn[b].alloc(N)))
      return st;
  cudaStream_t s = dem_stream(d);
  HG_CUDA_TRY(cudaMemsetAsync(d->status.p, 0, sizeof(uint32_t), s));
  HG_CUDA_TRY(cudaMemsetAsync(d->c_count.p, 0, 2 * sizeof(int32_t), s));
  d->bins = hg_dem::BINS_DIRTY;
  d->desc_valid = false;
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  return HG_OK;
}

hg_status dem_reset_history(hg_dem *d) {
  HG_CUDA_TRY(cudaMemsetAsync(d->c_count.p, 0, 2 * sizeof(int32_t), dem_stream(d)));
  d->history_valid = false;
  d->desc_valid = false;
  return HG_OK;
}

// The bodies' positions, radii, flags or number changed outside dem_step: the
// next step bins them anew.
void dem_bodies_changed(hg_dem *d) {
  d->bins = hg_dem::BINS_DIRTY;
}

hg_status dem_prepare(hg_dem *d, double dt) {
  if ((d->inv_valid && d->terms_dt == dt) || d->n == 0) return HG_OK;
  HG_LAUNCH(kd_body_terms, blocks_for(d->n, 256), 256, 0, dem_stream(d), d->n, dt, d->p.g[0],
            d->p.g[1], d->m0.p, d->I0.p, d->w.p, reinterpret_cast<double4 *>(d->minv.p));
  HG_CHECK_LAUNCH();
  d->inv_valid = true;
  d->terms_dt = dt;
  return HG_OK;
}

// The contact law's grid: one resident wave, so that the grid-stride loop runs
// no partial second wave.
void dem_set_launch_shapes(hg_dem *d) {
  int per_sm = 0;
  cudaError_t e = d->p.precision == HG_PRECISION_MIXED
                      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kdx_contacts,
                                                                      CONTACT_THREADS, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kd_contacts,
                                                                      CONTACT_THREADS, 0);
  if (e != cudaSuccess || per_sm < 1) {
    (void)cudaGetLastError();
    per_sm = 4;
  }
  d->contact_grid = d->ctx->num_sms * per_sm;
}

void dem_bin_args(const hg_dem *d, BinArgs *out) {
  BinArgs &H = *out;
  H.n = d->n;
  H.H = d->cell_h;
  H.invH = 1.0 / d->cell_h;
  // the hash table grows with the live body count (at most the capacity's)
  H.mask = (1u << table_bits(d->n)) - 1u;
  H.nplanes = d->p.nplanes;
  H.ndrums = d->p.ndrums;
  for (int k = 0; k < HG_MAX_DRUMS; ++k) {
    H.dx[k][0] = d->p.dx[k][0];
    H.dx[k][1] = d->p.dx[k][1];
    H.dr[k] = d->p.dr[k];
  }
  for (int k = 0; k < HG_MAX_PLANES; ++k)
    for (int c = 0; c < 2; ++c) {
      H.px[k][c] = d->p.px[k][c];
      H.pn[k][c] = d->p.pn[k][c];
      H.pxf[k][c] = (float)d->p.px[k][c];
      H.pnf[k][c] = (float)d->p.pn[k][c];
    }
  H.r = d->r.p;
  H.fixed = d->fixed.p;
  H.rec = d->brec.p;
  H.heads = d->heads.p;
  H.pc = d->pc.p;
  H.in_count = d->in_count.p;
  H.tiles = search_by_cells(d) ? d->tiles.p : nullptr;
  H.tile_shift = tile_shift_for(d->n);
}

void dem_binned(hg_dem *d) {
  if (d->bins == hg_dem::BINS_CLEAR) d->bins = hg_dem::BINS_FILLED;
}

hg_status dem_step(hg_dem *d, double dt, int weighted, bool bin_next, double *q_before) {
  cudaStream_t s = dem_stream(d);
  const int64_t n = d->n;
  if (n == 0) return HG_OK;
  hg_status st;
  if ((st = dem_prepare(d, dt))) return st;
  const int shift = tile_shift_for(n);
  const int ntiles = (int)(((n - 1) >> shift) + 1);
  const bool few = search_by_cells(d);
  BinArgs H;
  dem_bin_args(d, &H);
  const uint32_t mask = H.mask;
  const int bins = d->bins;
  d->bins = hg_dem::BINS_DIRTY; // until the step is queued
  if (bins == hg_dem::BINS_DIRTY) {
    HG_CUDA_TRY(cudaMemsetAsync(d->heads.p, 0xFF, sizeof(int32_t) * ((int64_t)d->mask + 1), s));
    HG_CUDA_TRY(cudaMemsetAsync(d->tiles.p, 0, sizeof(int32_t) * 4 * MAX_TILES, s));
  }
  if (bins != hg_dem::BINS_FILLED) {
    HG_LAUNCH_PDL(kd_bin, blocks_for(n, 128), 128, 0, s, H, d->q.p);
    HG_CHECK_LAUNCH();
  }
  const int nb = 1 - d->cc; // buffer receiving this step's contacts
  PairArgs A;
  A.n = n;
  A.mask = mask;
  A.rec = d->brec.p;
  A.Hf = (float)d->cell_h;
  A.tol = (float)(4.0e-6 * d->cell_h);
  A.heads = d->heads.p;
  A.q = d->q.p;
  A.r = d->r.p;
  A.nstatic = d->p.nplanes + d->p.ndrums;
  A.pc = d->pc.p;
  A.in_count = d->in_count.p;
  A.plist = d->plist.p;
  A.desc = d->desc[nb].p;
  A.descn = d->descn[nb].p;
  A.in_cursor = d->in_cursor.p;
  A.tiles = d->tiles.p;
  A.tile_shift = shift;
  A.ntiles = ntiles;
  A.add_tiles = few;
  A.keys = d->ckey[nb].p;
  A.ccap = d->ccap;
  A.count = d->c_count.p + nb;
  A.range = d->cc_range.p;
  A.status = d->status.p;
  if (few) {
    HG_LAUNCH_PDL(kd_pairs, blocks_for(5 * n, 128), 128, 0, s, A);
    HG_CHECK_LAUNCH();
    HG_LAUNCH_PDL(kd_pairs_emit<64>, blocks_for(n, 64), 64, 0, s, A);
  } else {
    HG_LAUNCH_PDL(kd_pairs_body, blocks_for(n, 128), 128, 0, s, A);
    HG_CHECK_LAUNCH();
    HG_LAUNCH_PDL(kd_tile_sums, ntiles, 256, 0, s, n, shift, d->pc.p, d->in_count.p, d->tiles.p);
    HG_CHECK_LAUNCH();
    HG_LAUNCH_PDL(kd_pairs_emit<256>, blocks_for(n, 256), 256, 0, s, A);
  }
  HG_CHECK_LAUNCH();
  ContactArgs Cg;
  Cg.n = n;
  Cg.dt = dt;
  Cg.weighted = weighted;
  Cg.kn = d->p.kn;
  Cg.kt = d->p.kt;
  Cg.gn = d->p.gn;
  Cg.gt = d->p.gt;
  Cg.mu = d->p.mu;
  Cg.half_gn = 0.5 * d->p.gn;
  Cg.half_gt = 0.5 * d->p.gt;
  Cg.mu2_32 = (float)(d->p.mu * d->p.mu);
  Cg.nplanes = d->p.nplanes;
  Cg.ndrums = d->p.ndrums;
  for (int k = 0; k < HG_MAX_DRUMS; ++k) {
    Cg.dx[k][0] = d->p.dx[k][0];
    Cg.dx[k][1] = d->p.dx[k][1];
    Cg.dr[k] = d->p.dr[k];
  }
  for (int k = 0; k < HG_MAX_PLANES; ++k)
    for (int c = 0; c < 2; ++c) {
      Cg.px[k][c] = d->p.px[k][c];
      Cg.pn[k][c] = d->p.pn[k][c];
    }
  Cg.q = d->q.p;
  Cg.v = d->v.p;
  Cg.r = d->r.p;
  Cg.w = d->w.p;
  Cg.count = d->c_count.p + nb;
  Cg.keys = d->ckey[nb].p;
  Cg.rec = d->crec[nb].p;
  Cg.load = d->load.p;
  Cg.desc = d->desc[nb].p;
  Cg.in_cursor = d->in_cursor.p;
  Cg.in_list = d->in_list.p;
  Cg.old_keys = d->ckey[d->cc].p;
  Cg.old_rec = d->crec[d->cc].p;
  Cg.old_count = d->c_count.p + d->cc;
  Cg.old_desc = d->desc_valid ? d->desc[d->cc].p : nullptr;
  Cg.old_descn = d->descn[d->cc].p;
  Cg.heads = d->heads.p;
  Cg.nheads = (int64_t)mask + 1;
  Cg.tiles = d->tiles.p;
  Cg.ccap = d->ccap;
  Cg.status = d->status.p;
  // one wave, or the CTAs that the contacts the buffers hold can fill
  const int64_t chunks = std::max<int64_t>((d->ccap + 31) / 32, (n + 31) / 32);
  const int cgrid = (int)std::min<int64_t>(d->contact_grid, chunks);
  if (d->p.precision == HG_PRECISION_MIXED)
    HG_LAUNCH_PDL(kdx_contacts, cgrid, CONTACT_THREADS, 0, s, Cg);
  else
    HG_LAUNCH_PDL(kd_contacts, cgrid, CONTACT_THREADS, 0, s, Cg);
  HG_CHECK_LAUNCH();
  IntegrateArgs I;
  I.n = n;
  I.ccap = d->ccap;
  I.dt = dt;
  I.q = d->q.p;
  I.v = d->v.p;
  I.q_before = q_before;
  I.terms = reinterpret_cast<const double4 *>(d->minv.p);
  I.fixed = d->fixed.p;
  I.desc = d->desc[nb].p;
  I.descn = d->descn[nb].p;
  I.in_cursor = d->in_cursor.p;
  I.in_list = d->in_list.p;
  I.load = d->load.p;
  I.keys = d->ckey[nb].p;
  I.range = d->cc_range.p;
  I.status = d->status.p;
  auto integrate = d->p.precision == HG_PRECISION_MIXED
                       ? (bin_next ? kdx_integrate<true> : kdx_integrate<false>)
                       : (bin_next ? kd_integrate<true> : kd_integrate<false>);
  // one warp per CTA spreads few bodies over all SMs' FP64 pipes
  const int it = few ? 32 : 128;
  HG_LAUNCH_PDL(integrate, blocks_for(n, it), it, 0, s, I, H);
  HG_CHECK_LAUNCH();
  d->cc = nb;
  d->history_valid = true;
  d->desc_valid = true;
  d->bins = bin_next ? hg_dem::BINS_FILLED : hg_dem::BINS_CLEAR;
  return HG_OK;
}

// ---- contact history after bodies are removed -------------------------------
//
// PenaltyImpactFrictionMap::deleteCacheEntries / relabelEntries
// (PenaltyImpactFrictionMap.cpp:1199-1278): contacts of removed bodies are
// dropped and the others renumbered. The map is monotone, so the list stays
// sorted by (kind, first, second) and a stable compaction keeps it valid for
// the next step's history lookup.
namespace {

__device__ __forceinline__ bool relabel_one(int64_t key, const int32_t *map, int64_t nmap,
                                            int64_t &out, int32_t &a2, int32_t &b2) {
  const int64_t kind = key >> 60;
  const int64_t a = (key >> 30) & 0x3FFFFFFF, b = key & 0x3FFFFFFF;
  a2 = a < nmap ? map[a] : -1;
  b2 = kind == 0 ? (int32_t)b : (b < nmap ? map[b] : -1); // kind 0: plane index
  out = (kind << 60) | ((int64_t)a2 << 30) | (int64_t)b2;
  return a2 >= 0 && b2 >= 0;
}

__global__ void kd_relabel_keep(int64_t ccap, const int32_t *__restrict__ count,
                                const int64_t *__restrict__ keys, const int32_t *__restrict__ map,
                                int64_t nmap, int32_t *keep) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k > ccap) return;
  const int64_t c = min((int64_t)*count, ccap);
  int64_t nk;
  int32_t a2, b2;
  keep[k] = (k < c && relabel_one(keys[k], map, nmap, nk, a2, b2)) ? 1 : 0;
}

__global__ void kd_relabel_move(int64_t ccap, const int32_t *__restrict__ count,
                                const int64_t *__restrict__ keys, const double *__restrict__ rec,
                                const int32_t *__restrict__ map, int64_t nmap,
                                const int32_t *__restrict__ off, int64_t *okeys, double *orec,
                                int32_t *ocount) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t c = min((int64_t)*count, ccap);
  if (k == 0) *ocount = off[c];
  if (k >= c) return;
  int64_t nk;
  int32_t a2, b2;
  if (!relabel_one(keys[k], map, nmap, nk, a2, b2)) return;
  const int64_t o = off[k];
  okeys[o] = nk;
  for (int j = 0; j < RW; ++j) orec[o * RW + j] = rec[k * RW + j];
  orec[o * RW + 1] = (double)a2;
  orec[o * RW + 2] = (double)b2;
}

} // namespace

hg_status dem_relabel_device(hg_dem *d, const int32_t *map, int64_t nmap) {
  if (!d->history_valid) return HG_OK;
  cudaStream_t s = dem_stream(d);
  const int64_t C = d->ccap;
  DevBuf<int32_t> keep, off, tmp;
  hg_status st;
  if ((st = keep.alloc(C + 1)) || (st = off.alloc(C + 1)) || (st = tmp.alloc(scan_tmp_size(C + 1))))
    return st;
  const int nb = 1 - d->cc;
  HG_LAUNCH(kd_relabel_keep, blocks_for(C + 1, 256), 256, 0, s, C, d->c_count.p + d->cc,
            d->ckey[d->cc].p, map, nmap, keep.p);
  HG_CHECK_LAUNCH();
  if ((st = exclusive_scan_i32(keep.p, off.p, C + 1, tmp.p, s))) return st;
  HG_LAUNCH(kd_relabel_move, blocks_for(C + 1, 256), 256, 0, s, C, d->c_count.p + d->cc,
            d->ckey[d->cc].p, d->crec[d->cc].p, map, nmap, off.p, d->ckey[nb].p,
            d->crec[nb].p, d->c_count.p + nb);
  HG_CHECK_LAUNCH();
  d->cc = nb;
  d->desc_valid = false; // the bodies' lists moved
  return HG_OK;
}

hg_status dem_relabel(hg_dem *d, const int32_t *map_host, int64_t nmap) {
  if (!d->history_valid) return HG_OK;
  cudaStream_t s = dem_stream(d);
  DevBuf<int32_t> map;
  hg_status st;
  if ((st = map.alloc(std::max<int64_t>(nmap, 1)))) return st;
  if (nmap > 0)
    HG_CUDA_TRY(cudaMemcpyAsync(map.p, map_host, sizeof(int32_t) * nmap, cudaMemcpyHostToDevice, s));
  if ((st = dem_relabel_device(d, map.p, nmap))) return st;
  // the map was copied from the caller's memory: it may go once this returns
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  return HG_OK;
}

namespace {

// Moves kept bodies to their new slots (old_to_new, monotone) in scratch
// arrays; the caller copies the scratch back.
__global__ void kd_compact_bodies(int64_t n_old, const int32_t *__restrict__ map,
                                  const double *__restrict__ q, const double *__restrict__ v,
                                  const double *__restrict__ r, const double *__restrict__ m0,
                                  const double *__restrict__ I0, const double *__restrict__ w,
                                  const uint8_t *__restrict__ fixed, double *tq, double *tv,
                                  double *tr, double *tm, double *tI, double *tw, uint8_t *tf) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n_old) return;
  const int32_t j = map[i];
  if (j < 0) return;
  for (int c = 0; c < 3; ++c) {
    tq[3 * (int64_t)j + c] = q[3 * i + c];
    tv[3 * (int64_t)j + c] = v[3 * i + c];
  }
  tr[j] = r[i];
  tm[j] = m0[i];
  tI[j] = I0[i];
  tw[j] = w[i];
  tf[j] = fixed[i];
}

__global__ void kd_ones(double *a, int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) a[i] = 1.0;
}

} // namespace

hg_status dem_edit(hg_dem *d, int64_t n_old, const int32_t *map_host, int64_t n_keep,
                   int64_t n_add, const double *q, const double *v, const double *r,
                   const double *m, const double *I, const uint8_t *fixed) {
  cudaStream_t s = dem_stream(d);
  hg_status st;
  DevBuf<int32_t> map;
  if (n_old > 0) {
    DevBuf<double> tq, tv, tr, tm, tI, tw;
    DevBuf<uint8_t> tf;
    const int64_t k = std::max<int64_t>(n_keep, 1);
    if ((st = map.alloc(n_old)) || (st = tq.alloc(3 * k)) || (st = tv.alloc(3 * k)) ||
        (st = tr.alloc(k)) || (st = tm.alloc(k)) || (st = tI.alloc(k)) || (st = tw.alloc(k)) ||
        (st = tf.alloc(k)))
      return st;
    HG_CUDA_TRY(cudaMemcpyAsync(map.p, map_host, sizeof(int32_t) * n_old, cudaMemcpyHostToDevice, s));
    HG_LAUNCH(kd_compact_bodies, blocks_for(n_old, 256), 256, 0, s, n_old, map.p, d->q.p, d->v.p,
              d->r.p, d->m0.p, d->I0.p, d->w.p, d->fixed.p, tq.p, tv.p, tr.p, tm.p, tI.p, tw.p,
              tf.p);
    HG_CHECK_LAUNCH();
    if (n_keep > 0) {
      HG_CUDA_TRY(cudaMemcpyAsync(d->q.p, tq.p, sizeof(double) * 3 * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->v.p, tv.p, sizeof(double) * 3 * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->r.p, tr.p, sizeof(double) * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->m0.p, tm.p, sizeof(double) * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->I0.p, tI.p, sizeof(double) * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->w.p, tw.p, sizeof(double) * n_keep, cudaMemcpyDeviceToDevice, s));
      HG_CUDA_TRY(cudaMemcpyAsync(d->fixed.p, tf.p, n_keep, cudaMemcpyDeviceToDevice, s));
    }
    if ((st = dem_relabel_device(d, map.p, n_old))) return st;
  }
  if (n_add > 0) {
    const int64_t o = n_keep;
    HG_CUDA_TRY(cudaMemcpyAsync(d->q.p + 3 * o, q, sizeof(double) * 3 * n_add, cudaMemcpyHostToDevice, s));
    HG_CUDA_TRY(cudaMemcpyAsync(d->v.p + 3 * o, v, sizeof(double) * 3 * n_add, cudaMemcpyHostToDevice, s));
    HG_CUDA_TRY(cudaMemcpyAsync(d->r.p + o, r, sizeof(double) * n_add, cudaMemcpyHostToDevice, s));
    HG_CUDA_TRY(cudaMemcpyAsync(d->m0.p + o, m, sizeof(double) * n_add, cudaMemcpyHostToDevice, s));
    HG_CUDA_TRY(cudaMemcpyAsync(d->I0.p + o, I, sizeof(double) * n_add, cudaMemcpyHostToDevice, s));
    if (fixed) {
      HG_CUDA_TRY(cudaMemcpyAsync(d->fixed.p + o, fixed, n_add, cudaMemcpyHostToDevice, s));
    } else {
      HG_CUDA_TRY(cudaMemsetAsync(d->fixed.p + o, 0, n_add, s));
    }
    HG_LAUNCH(kd_ones, blocks_for(n_add, 256), 256, 0, s, d->w.p + o, n_add);
    HG_CHECK_LAUNCH();
  }
  d->n = n_keep + n_add;
  d->inv_valid = false;
  d->desc_valid = false;
  dem_bodies_changed(d);
  return HG_OK;
}


hg_status dem_download_contacts(hg_dem *d, int64_t cap, double *rec, int64_t *count) {
  cudaStream_t s = dem_stream(d);
  int32_t c = 0;
  if (d->history_valid) {
    HG_CUDA_TRY(cudaMemcpyAsync(&c, d->c_count.p + d->cc, sizeof(int32_t),
                                cudaMemcpyDeviceToHost, s));
    HG_CUDA_TRY(cudaStreamSynchronize(s));
  }
  const int64_t total = std::min<int64_t>(c, d->ccap);
  *count = total;
  const int64_t k = std::min<int64_t>(total, cap);
  if (k > 0) {
    HG_CUDA_TRY(cudaMemcpyAsync(rec, d->crec[d->cc].p, sizeof(double) * RW * k,
                                cudaMemcpyDeviceToHost, s));
    HG_CUDA_TRY(cudaStreamSynchronize(s));
    // drum contacts are static objects after the planes on the device; the
    // export names them by kind and drum index
    if (d->p.ndrums > 0)
      for (int64_t i = 0; i < k; ++i) {
        double *o = rec + i * RW;
        if (o[0] == (double)K_PLANE && o[2] >= (double)d->p.nplanes) {
          o[0] = (double)HG_DEM_KIND_DRUM;
          o[2] -= (double)d->p.nplanes;
        }
      }
  }
  return HG_OK;
}

hg_status dem_candidate_pairs(hg_context *ctx, int64_t n, const double *mn, const double *mx,
                              int64_t cap, int32_t *pairs, int64_t *count) {
  cudaStream_t s = ctx->stream;
  *count = 0;
  if (n == 0) return HG_OK;
  double H = 0.0, amax = 0.0;
  for (int64_t i = 0; i < 2 * n; ++i) {
    H = std::max(H, mx[i] - mn[i]);
    amax = std::max(amax, std::max(std::fabs(mn[i]), std::fabs(mx[i])));
  }
  H = H * (1.0 + 1.0e-6);
  if (amax / H > 1.0e9) return fail(HG_ERR_INVALID_ARGUMENT, "boxes too small for their coordinates");
  const uint32_t bits = table_bits(n);
  const int64_t T = (int64_t)1 << bits;
  DevBuf<double> dmn, dmx;
  DevBuf<int2> home;
  DevBuf<int32_t> bcount, bstart, bcursor, items, cnt, off, tmp, dpairs;
  DevBuf<uint32_t> status;
  hg_status st;
  if ((st = dmn.alloc(2 * n)) || (st = dmx.alloc(2 * n)) || (st = home.alloc(n)) ||
      (st = bcount.alloc(T)) || (st = bstart.alloc(T)) || (st = bcursor.alloc(T)) ||
      (st = items.alloc(n)) || (st = cnt.alloc(n + 1)) || (st = off.alloc(n + 1)) ||
      (st = tmp.alloc(std::max(scan_tmp_size(T), scan_tmp_size(n + 1)))) ||
      (st = status.alloc(1)))
    return st;
  HG_CUDA_TRY(cudaMemcpyAsync(dmn.p, mn, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, s));
  HG_CUDA_TRY(cudaMemcpyAsync(dmx.p, mx, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, s));
  HG_CUDA_TRY(cudaMemsetAsync(status.p, 0, sizeof(uint32_t), s));
  HG_CUDA_TRY(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * (n + 1), s));
  BroadArgs B;
  B.n = n;
  B.H = H;
  B.mask = (uint32_t)(T - 1);
  B.mn = dmn.p;
  B.mx = dmx.p;
  if ((st = build_buckets(s, B, bcount.p, bstart.p, bcursor.p, items.p, home.p, tmp.p))) return st;
  HG_LAUNCH(kd_box_pairs<false>, blocks_for(n, 128), 128, 0, s, B, home.p, bstart.p, bcount.p,
            items.p, cnt.p, off.p, nullptr, 0, status.p);
  HG_CHECK_LAUNCH();
  if ((st = exclusive_scan_i32(cnt.p, off.p, n + 1, tmp.p, s))) return st;
  int32_t total = 0;
  uint32_t word = 0;
  HG_CUDA_TRY(cudaMemcpyAsync(&total, off.p + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaMemcpyAsync(&word, status.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  if (word & HG_STATUS_CELL_OVERFLOW)
    return fail(HG_ERR_CAPACITY, "more than 32 overlapping boxes for one box");
  if ((st = dpairs.alloc(2 * (int64_t)std::max<int32_t>(total, 1)))) return st;
  HG_LAUNCH(kd_box_pairs<true>, blocks_for(n, 128), 128, 0, s, B, home.p, bstart.p, bcount.p,
            items.p, cnt.p, off.p, dpairs.p, (int64_t)total, status.p);
  HG_CHECK_LAUNCH();
  const int64_t k = std::min<int64_t>(total, cap);
  if (k > 0)
    HG_CUDA_TRY(cudaMemcpyAsync(pairs, dpairs.p, sizeof(int32_t) * 2 * k, cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  *count = total;
  return HG_OK;
}

} // namespace hg

// ---- allocation-free candidate-pair search -------------------------------------
//
// The same broadphase as hg_dem_candidate_pairs, with every device temporary
// placed in one file-scope __device__ array instead of cudaMalloc'd buffers.

namespace hg {
namespace {

constexpr int64_t SP_MAX_BOXES = HG_STATIC_PAIRS_MAX_BOXES;
constexpr int64_t SP_MAX_PAIRS = HG_STATIC_PAIRS_MAX_PAIRS;
constexpr uint32_t SP_TABLE_BITS = 15; // 32768 buckets >= 2 * SP_MAX_BOXES
constexpr int64_t SP_TABLE = (int64_t)1 << SP_TABLE_BITS;
static_assert(SP_TABLE >= 2 * SP_MAX_BOXES, "hash table too small");

constexpr size_t sp_align(size_t b) { return (b + 255) & ~(size_t)255; }
// Byte offsets of the regions inside the scratch array.
constexpr size_t SP_MN = 0;
constexpr size_t SP_MX = SP_MN + sp_align(sizeof(double) * 2 * SP_MAX_BOXES);
constexpr size_t SP_HOME = SP_MX + sp_align(sizeof(double) * 2 * SP_MAX_BOXES);
constexpr size_t SP_BCOUNT = SP_HOME + sp_align(sizeof(int2) * SP_MAX_BOXES);
constexpr size_t SP_BSTART = SP_BCOUNT + sp_align(sizeof(int32_t) * SP_TABLE);
constexpr size_t SP_BCURSOR = SP_BSTART + sp_align(sizeof(int32_t) * SP_TABLE);
constexpr size_t SP_ITEMS = SP_BCURSOR + sp_align(sizeof(int32_t) * SP_TABLE);
constexpr size_t SP_CNT = SP_ITEMS + sp_align(sizeof(int32_t) * SP_MAX_BOXES);
constexpr size_t SP_OFF = SP_CNT + sp_align(sizeof(int32_t) * (SP_MAX_BOXES + 1));
constexpr size_t SP_TMP = SP_OFF + sp_align(sizeof(int32_t) * (SP_MAX_BOXES + 1));
// the scans run over the bucket table and over the per-box counts
constexpr size_t SP_TMP_INTS = 256;
static_assert(SP_TMP_INTS >= (size_t)scan_tmp_size(SP_TABLE > SP_MAX_BOXES + 1 ? SP_TABLE
                                                                             : SP_MAX_BOXES + 1),
              "scan scratch region too small for the largest scan");
constexpr size_t SP_PAIRS = SP_TMP + sp_align(sizeof(int32_t) * SP_TMP_INTS);
constexpr size_t SP_STATUS = SP_PAIRS + sp_align(sizeof(int32_t) * 2 * SP_MAX_PAIRS);
constexpr size_t SP_BYTES = SP_STATUS + 256;

} // namespace
} // namespace hg

// Every GPU that loads the library holds this array (about 3.4 MB) until the
// process exits. Host code must not pass its name to a kernel: on the host
// the name is a stand-in, not a device address; the device address comes from
// cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_pairs_scratch[hg::SP_BYTES];

namespace hg {
namespace {

std::mutex g_sp_mutex;
unsigned char *g_sp_ptr[256] = {};

// Device address of g_pairs_scratch on the current device, looked up once per
// device (the lookup initialises the module on that device). The address is
// kept for the life of the process: a cudaDeviceReset of the device unloads
// the module and ends every context of this library on it, this address
// included, so no call may follow a reset.
hg_status static_scratch(int device, unsigned char **out) {
  if (device < 0 || device >= 256) return fail(HG_ERR_INVALID_ARGUMENT, "device index out of range");
  std::lock_guard<std::mutex> lock(g_sp_mutex);
  if (!g_sp_ptr[device]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_pairs_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_pairs_scratch)");
    g_sp_ptr[device] = static_cast<unsigned char *>(p);
  }
  *out = g_sp_ptr[device];
  return HG_OK;
}

} // namespace
} // namespace hg

extern "C" hg_status hg_dem_candidate_pairs_static(hg_context *ctx, int64_t n,
                                                   const double *aabb_min,
                                                   const double *aabb_max, int64_t cap,
                                                   int32_t *pairs, int64_t *count) {
  using namespace hg;
  if (!ctx || !count || n < 0 || (n > 0 && (!aabb_min || !aabb_max)) || (cap > 0 && !pairs) ||
      cap < 0)
    return fail(HG_ERR_INVALID_ARGUMENT, "bad argument");
  if (n > SP_MAX_BOXES)
    return fail(HG_ERR_CAPACITY, "hg_dem_candidate_pairs_static takes at most " +
                                     std::to_string(SP_MAX_BOXES) + " boxes, got " +
                                     std::to_string(n));
  *count = 0;
  double H = 0.0, amax = 0.0;
  for (int64_t i = 0; i < 2 * n; ++i) {
    if (!std::isfinite(aabb_min[i]) || !std::isfinite(aabb_max[i]) || !(aabb_min[i] < aabb_max[i]))
      return fail(HG_ERR_INVALID_ARGUMENT, "boxes must be finite with min < max");
    H = std::max(H, aabb_max[i] - aabb_min[i]);
    amax = std::max(amax, std::max(std::fabs(aabb_min[i]), std::fabs(aabb_max[i])));
  }
  if (n == 0) return HG_OK;
  H = H * (1.0 + 1.0e-6);
  if (amax / H > 1.0e9) return fail(HG_ERR_INVALID_ARGUMENT, "boxes too small for their coordinates");
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != ctx->device) cudaSetDevice(ctx->device);
  struct Restore {
    int dev;
    ~Restore() {
      if (dev >= 0) cudaSetDevice(dev);
    }
  } restore{prev != ctx->device ? prev : -1};
  unsigned char *base = nullptr;
  hg_status st = static_scratch(ctx->device, &base);
  if (st != HG_OK) return st;
  cudaStream_t s = ctx->stream;
  double *dmn = reinterpret_cast<double *>(base + SP_MN);
  double *dmx = reinterpret_cast<double *>(base + SP_MX);
  int2 *home = reinterpret_cast<int2 *>(base + SP_HOME);
  int32_t *bcount = reinterpret_cast<int32_t *>(base + SP_BCOUNT);
  int32_t *bstart = reinterpret_cast<int32_t *>(base + SP_BSTART);
  int32_t *bcursor = reinterpret_cast<int32_t *>(base + SP_BCURSOR);
  int32_t *items = reinterpret_cast<int32_t *>(base + SP_ITEMS);
  int32_t *cnt = reinterpret_cast<int32_t *>(base + SP_CNT);
  int32_t *off = reinterpret_cast<int32_t *>(base + SP_OFF);
  int32_t *tmp = reinterpret_cast<int32_t *>(base + SP_TMP);
  int32_t *dpairs = reinterpret_cast<int32_t *>(base + SP_PAIRS);
  uint32_t *status = reinterpret_cast<uint32_t *>(base + SP_STATUS);
  // Inputs in, counters cleared: the array keeps the previous call's contents.
  HG_CUDA_TRY(cudaMemcpyAsync(dmn, aabb_min, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, s));
  HG_CUDA_TRY(cudaMemcpyAsync(dmx, aabb_max, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, s));
  HG_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(uint32_t), s));
  HG_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (n + 1), s));
  const uint32_t bits = std::min<uint32_t>(table_bits(n), SP_TABLE_BITS);
  BroadArgs B;
  B.n = n;
  B.H = H;
  B.mask = (1u << bits) - 1u;
  B.mn = dmn;
  B.mx = dmx;
  if ((st = build_buckets(s, B, bcount, bstart, bcursor, items, home, tmp))) return st;
  HG_LAUNCH(kd_box_pairs<false>, blocks_for(n, 128), 128, 0, s, B, home, bstart, bcount, items,
            cnt, off, nullptr, 0, status);
  HG_CHECK_LAUNCH();
  if ((st = exclusive_scan_i32(cnt, off, n + 1, tmp, s))) return st;
  int32_t total = 0;
  uint32_t word = 0;
  HG_CUDA_TRY(cudaMemcpyAsync(&total, off + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaMemcpyAsync(&word, status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  if (word & HG_STATUS_CELL_OVERFLOW)
    return fail(HG_ERR_CAPACITY, "more than 32 overlapping boxes for one box");
  if (total > SP_MAX_PAIRS)
    return fail(HG_ERR_CAPACITY, "hg_dem_candidate_pairs_static holds at most " +
                                     std::to_string(SP_MAX_PAIRS) + " pairs, found " +
                                     std::to_string(total));
  HG_LAUNCH(kd_box_pairs<true>, blocks_for(n, 128), 128, 0, s, B, home, bstart, bcount, items,
            cnt, off, dpairs, (int64_t)total, status);
  HG_CHECK_LAUNCH();
  const int64_t k = std::min<int64_t>(total, cap);
  if (k > 0)
    HG_CUDA_TRY(cudaMemcpyAsync(pairs, dpairs, sizeof(int32_t) * 2 * k, cudaMemcpyDeviceToHost, s));
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  *count = total;
  return HG_OK;
}
