// Node-node hybrid coupling (hybridgrains2dnew/Coupling.cpp,
// HybridGrains2DSim.cpp:116-220) over the FP64 MPM path and the DEM path.
//
// Compiled with --fmad=false. Grain-to-grid scatters use FP64 atomics (sums
// differ from the serial reference in order only); the packed grain and node
// lists are built with a scan, so they keep the reference's stable-partition
// order (Coupling.cpp:113-127). With a MIXED (FP32) MPM bulk the grains' and
// contacts' stencil weights are FP32 over the same FP64 stencils; the grids
// and the exchange stay FP64. The kernels are bound by the FP64 pipe and by
// the chain of launches: stencils are formed as in mpm_axis.cuh, a grain's are
// shared by what it does at one position, few grains go to one-warp CTAs (a
// CTA on every SM), and each grid is cleared by the kernel that last reads it.
// Per step of the hybrid column (9,000 grains on 100,000 points), with eight
// launches, four memsets and a copy before: MIXED bulk 128 -> 69 us, FP64 bulk
// (its MPM kernels included) 367 -> 201 us.
//
// Kernels:
//   kc_grain_scatter  rasterizeGrainMass (Coupling.cpp:22-140) and
//                     rasterizeGrainMom (Coupling.cpp:287-363), after the DEM
//                     step: both are taken at the positions before it, and the
//                     nodes' MPM mass does not change in between
//   kc_flag_nodes /   std::stable_partition of grains and nodes
//   kc_pack             (Coupling.cpp:113-127)
//   kc_update_nodes   updateVelocitiesOnGrid (Coupling.cpp:533-579) and the
//                     homog_factor loop (HybridGrains2DSim.cpp:183-197), over
//                     every node
//   kc_transfer       transferToGrain, FLIP with alpha = 1 (Coupling.cpp:
//                     468-527), updatePositions_node_node (Coupling.cpp:
//                     581-591), then the scatter of
//                     ResamplingTools::homogenizeVelocity
//                     (ResamplingTools.cpp:830-884), and the binning for the
//                     next DEM step
//   kc_homogenize     the rest of homogenizeVelocity over the nodes, and
//                     ResamplingTools::homogenizeStress (ResamplingTools.cpp:
//                     744-813) over the contacts
#include "hg_internal.cuh"
#include "mpm_basis.cuh"
#include "mpm_axis.cuh"
#include "dem_bins.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

namespace hg {

namespace {

struct GridGeom {
  int nx, ny;
  double gx, gy, h;
  double inv_h;
};

GridGeom geom(const hg_mpm *m) {
  return GridGeom{m->p.nx, m->p.ny, m->p.gmin[0], m->p.gmin[1], m->p.h, m->p.inv_h};
}

__device__ __forceinline__ bool node_ok(const GridGeom &G, int ix, int iy) {
  return ix >= 0 && iy >= 0 && ix <= G.nx && iy <= G.ny;
}

// FP32 1-D weights (a MIXED bulk) of LinearBasisFunctions.cpp:6-13 and
// uGIMPLinearBasisFunctions.cpp:6-22 in units of the cell width (for uGIMP,
// L(d) with a = hl / h: (1 + a - d)^2 / 2, 2a (1 - d) or 2a - (a^2 + d^2)
// by band).
template <int BASIS> __device__ __forceinline__ float weight1d32(float d, float a) {
  const float dd = fabsf(d);
  if (BASIS == HG_BASIS_LINEAR) return dd < 1.0f ? 1.0f - dd : 0.0f;
  if (dd >= 1.0f + a) return 0.0f;
  if (dd >= 1.0f - a) return 0.5f * (1.0f + a - dd) * (1.0f + a - dd);
  if (dd >= a) return 2.0f * a * (1.0f - dd);
  return 2.0f * a - (a * a + dd * dd);
}

// The stencil of a position with half-width hl: the reference's FP64 node
// range, and the 2-D weights as products of per-axis factors, FP32 (W32, a
// MIXED bulk) or FP64. In FP32 the offset from the stencil's first node, in
// cell widths, is formed in FP64 and rounded once.
template <int BASIS, bool W32> struct GridStencil {
  int x0, y0, nx, ny;
  double ax[W32 ? 1 : STENCIL_AXIS], ay[W32 ? 1 : STENCIL_AXIS];
  float fx[W32 ? STENCIL_AXIS : 1], fy[W32 ? STENCIL_AXIS : 1];

  __device__ __forceinline__ bool wide() const { return nx > STENCIL_AXIS || ny > STENCIL_AXIS; }

  __device__ __forceinline__ void range(const GridGeom &G, double x, double y, double hl) {
    const Divisor H = divisor(G.h, G.inv_h);
    bool ok = H.ok;
    Axis<BASIS> X, Y;
    X.template range<false>(x, hl, G.gx, H, ok);
    Y.template range<false>(y, hl, G.gy, H, ok);
    x0 = X.i0;
    nx = X.n;
    y0 = Y.i0;
    ny = Y.n;
    if (!ok) {
      int x1, y1;
      stencil64(BASIS, x, y, hl, G.gx, G.gy, G.h, x0, y0, x1, y1);
      nx = x1 - x0 + 1;
      ny = y1 - y0 + 1;
    }
  }
  __device__ __forceinline__ void weights(const GridGeom &G, double x, double y, double hl) {
    if (W32) {
      const float ox = narrow((x - G.gx) * G.inv_h - (x0 >= 0 ? index_f64(x0) : (double)x0));
      const float oy = narrow((y - G.gy) * G.inv_h - (y0 >= 0 ? index_f64(y0) : (double)y0));
      const float a = narrow(hl * G.inv_h);
      const float norm = BASIS == HG_BASIS_LINEAR ? 1.0f : 1.0f / (4.0f * a * a);
#pragma unroll
      for (int k = 0; k < STENCIL_AXIS; ++k) {
        fx[k] = k < nx ? weight1d32<BASIS>(ox - (float)k, a) : 0.0f;
        fy[k] = k < ny ? weight1d32<BASIS>(oy - (float)k, a) * norm : 0.0f;
      }
      return;
    }
    const Divisor H = divisor(G.h, G.inv_h);
    bool ok = H.ok;
    Axis<BASIS> X, Y;
    X.i0 = x0;
    X.n = nx;
    Y.i0 = y0;
    Y.n = ny;
    if constexpr (BASIS == HG_BASIS_LINEAR) {
      X.template factors<false, false>(x, G.gx, H, ok);
      Y.template factors<false, false>(y, G.gy, H, ok);
      if (!ok) {
        X.template factors<false, true>(x, G.gx, H, ok);
        Y.template factors<false, true>(y, G.gy, H, ok);
      }
    } else {
      Extent E;
      E.set(hl, H);
      X.template factors<false>(x, E, G.gx, H);
      Y.template factors<false>(y, E, G.gy, H);
    }
    const double inv = BASIS == HG_BASIS_LINEAR ? 1.0 : 1.0 / (4.0 * hl * hl);
#pragma unroll
    for (int k = 0; k < (BASIS == HG_BASIS_LINEAR ? 2 : STENCIL_AXIS); ++k) {
      ax[k] = X.w[k];
      ay[k] = BASIS == HG_BASIS_LINEAR ? Y.w[k] : Y.w[k] * inv;
    }
  }
  // f(node, weight) over the nodes on the grid, y outer, x inner
  template <class F> __device__ __forceinline__ void each(const GridGeom &G, F &&f) const {
    constexpr int N = BASIS == HG_BASIS_LINEAR ? 2 : STENCIL_AXIS;
#pragma unroll
    for (int ky = 0; ky < N; ++ky) {
      if (ky >= ny) break;
#pragma unroll
      for (int kx = 0; kx < N; ++kx) {
        if (kx >= nx) break;
        if (!node_ok(G, x0 + kx, y0 + ky)) continue;
        const double w = W32 ? widen_f32(fx[kx] * fy[ky]) : ax[kx] * ay[ky];
        f((int64_t)(y0 + ky) * (G.nx + 1) + x0 + kx, w);
      }
    }
  }
  // the same with a stencil wider than the kernels hold, node by node
  template <class F>
  __device__ __forceinline__ void each_wide(const GridGeom &G, double x, double y, double hl,
                                            F &&f) const {
    for (int iy = y0; iy < y0 + ny; ++iy)
      for (int ix = x0; ix < x0 + nx; ++ix)
        if (node_ok(G, ix, iy))
          f((int64_t)iy * (G.nx + 1) + ix, weight64(BASIS, x, y, hl, ix, iy, G.gx, G.gy, G.h));
  }
};

// weights and visit in one, either form
template <int BASIS, bool W32, class F>
__device__ __forceinline__ void visit(GridStencil<BASIS, W32> &S, const GridGeom &G, double x,
                                      double y, double hl, F &&f) {
  if (S.wide()) {
    S.each_wide(G, x, y, hl, f);
    return;
  }
  S.weights(G, x, y, hl);
  S.each(G, f);
}

// a coupled node's MPM mass is not below or at 1e-6 (Coupling.cpp:22-140),
// compared as bit patterns; 1e-6f is the largest float not above it
__device__ __forceinline__ bool massive(float m) {
  return __float_as_int(m) > __float_as_int(1.0e-6f);
}
__device__ __forceinline__ bool massive(double m) {
  return __double_as_longlong(m) > __double_as_longlong(1.0e-6);
}

struct GrainArgs {
  GridGeom G;
  int64_t nb;
  const double *pos; // 3 per grain: the positions before the DEM step
  const double *hl0; // points.hl(0): the first material point's extent
  const uint8_t *fixed;
  const double *m0, *w;
  double *v, *q;
  int32_t *coupled;
};

// M: the MPM node mass type (double for an FP64 object, float for MIXED,
// where it is the P2G sum of this step before the grid update).
template <int BASIS, bool W32, typename M>
__global__ void kc_grain_scatter(const __grid_constant__ GrainArgs A, const M *g_mass,
                                 double *dem_mass, double *dem_mom) {
  pdl_wait();
  pdl_trigger();
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b >= A.nb) return;
  const GridGeom &G = A.G;
  bool all = !A.fixed[b];
  const double x = A.pos[3 * b], y = A.pos[3 * b + 1], hl = *A.hl0;
  GridStencil<BASIS, W32> S;
  if (all) {
    S.range(G, x, y, hl);
    constexpr int N = BASIS == HG_BASIS_LINEAR ? 2 : STENCIL_AXIS;
    if (S.wide()) {
      for (int iy = S.y0; iy < S.y0 + S.ny; ++iy)
        for (int ix = S.x0; ix < S.x0 + S.nx; ++ix)
          if (node_ok(G, ix, iy) && !massive(g_mass[(int64_t)iy * (G.nx + 1) + ix])) all = false;
    } else {
      // (unrolled: the masses are loaded together)
#pragma unroll
      for (int ky = 0; ky < N; ++ky)
#pragma unroll
        for (int kx = 0; kx < N; ++kx) {
          const int ix = S.x0 + kx, iy = S.y0 + ky;
          if (kx < S.nx && ky < S.ny && node_ok(G, ix, iy))
            all &= massive(g_mass[(int64_t)iy * (G.nx + 1) + ix]);
        }
    }
  }
  A.coupled[b] = all ? 1 : 0;
  if (!all) return;
  const double pm = A.m0[b] * A.w[b]; // RigidBody2DState::getTotalMass
  const double px = pm * A.v[3 * b], py = pm * A.v[3 * b + 1];
  visit(S, G, x, y, hl, [&](int64_t i, double wt) {
    atomicAdd(&dem_mass[i], wt * pm);
    atomicAdd(&dem_mom[2 * i], wt * px);
    atomicAdd(&dem_mom[2 * i + 1], wt * py);
  });
}

__global__ void kc_flag_nodes(int64_t nn, const double *__restrict__ dem_mass, int32_t *flag) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nn) return;
  flag[i] = dem_mass[i] > 0.0 ? 1 : 0;
}

// Stable partition: writes the indices with flag set, in index order.
__global__ void kc_pack(int64_t n, const int32_t *__restrict__ flag,
                        const int32_t *__restrict__ pos, int32_t *out, int32_t *count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i > n) return;
  if (i == n) {
    *count = pos[n];
    return;
  }
  if (flag[i]) out[pos[i]] = (int32_t)i;
}

struct NodeArgs {
  int64_t nn;
  const double *dem_mass, *dem_mom;
  double *old_mass, *old_mom; // the previous step's, cleared here
  double *v_after, *a_after, *homog;
};

// Every node: its homogenisation factor (HybridGrains2DSim.cpp:183-197: 1/2
// where the DEM has mass, else 1 where the MPM has), and on the coupled nodes
// (DEM mass > 0) updateVelocitiesOnGrid; v_after and a_after are zero
// elsewhere. Nodes that were coupled in the previous step (its DEM mass is in
// the other set of grids) are the ones to zero and to clear for the next.
__device__ __forceinline__ bool coupled_node(const NodeArgs &A, int64_t i, double m_mpm,
                                             double &m_dem) {
  m_dem = A.dem_mass[i];
  const bool on = m_dem > 0.0, was = !f64_zero(A.old_mass[i]);
  A.homog[i] = on ? 0.5 : (m_mpm > 0.0 ? 1.0 : 0.0);
  if (was) {
    A.old_mass[i] = 0.0;
    reinterpret_cast<double2 *>(A.old_mom)[i] = make_double2(0.0, 0.0);
    if (!on) {
      reinterpret_cast<double2 *>(A.v_after)[i] = make_double2(0.0, 0.0);
      reinterpret_cast<double2 *>(A.a_after)[i] = make_double2(0.0, 0.0);
    }
  }
  return on;
}

__global__ void kc_update_nodes(const __grid_constant__ NodeArgs A,
                                const double *g_mass, double *g_mom_new) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.nn) return;
  const double m_mpm = g_mass[i];
  double m_dem;
  if (!coupled_node(A, i, m_mpm, m_dem)) return;
  double2 *mom = reinterpret_cast<double2 *>(g_mom_new);
  double2 p = mom[i];
  const double2 pd = reinterpret_cast<const double2 *>(A.dem_mom)[i];
  const Divisor S = divisor(m_mpm + m_dem), D = divisor(m_dem);
  const double lx = quot(m_dem * p.x - m_mpm * pd.x, S);
  const double ly = quot(m_dem * p.y - m_mpm * pd.y, S);
  p.x -= lx;
  p.y -= ly;
  mom[i] = p;
  reinterpret_cast<double2 *>(A.v_after)[i] = make_double2(quot(pd.x + lx, D), quot(pd.y + ly, D));
  reinterpret_cast<double2 *>(A.a_after)[i] = make_double2(quot(lx, D), quot(ly, D));
}

// updateVelocitiesOnGrid (Coupling.cpp:533-579) on a MIXED grid: the MPM
// node momentum after the grid update is gm v (FP32 velocity and mass), the
// exchange lambda is formed in FP64 as in kc_update_nodes, and the node's
// velocity and acceleration (va: v, a) take p_new - lambda; the acceleration
// (p_new - p) / (m dt) loses lambda / (m dt). Nodes without MPM mass keep
// their zero velocity, as (p_new = 0) / m is never formed for them.
__global__ void kc_update_nodes_x(const __grid_constant__ NodeArgs A, const float *gm,
                                  double dt, float4 *va) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.nn) return;
  const double m_mpm = widen_f32(gm[i]);
  double m_dem;
  if (!coupled_node(A, i, m_mpm, m_dem)) return;
  float4 g = va[i];
  const double2 pd = reinterpret_cast<const double2 *>(A.dem_mom)[i];
  const double px = m_mpm * widen_f32(g.x), py = m_mpm * widen_f32(g.y);
  const Divisor S = divisor(m_mpm + m_dem), D = divisor(m_dem);
  const double lx = quot(m_dem * px - m_mpm * pd.x, S);
  const double ly = quot(m_dem * py - m_mpm * pd.y, S);
  if (m_mpm > 0.0) {
    const Divisor M = divisor(m_mpm), T = divisor(m_mpm * dt);
    g.x = narrow(quot(px - lx, M));
    g.y = narrow(quot(py - ly, M));
    g.z = narrow(widen_f32(g.z) - quot(lx, T));
    g.w = narrow(widen_f32(g.w) - quot(ly, T));
    va[i] = g;
  }
  reinterpret_cast<double2 *>(A.v_after)[i] = make_double2(quot(pd.x + lx, D), quot(pd.y + ly, D));
  reinterpret_cast<double2 *>(A.a_after)[i] = make_double2(quot(lx, D), quot(ly, D));
}

__global__ void kc_set_scalar(double *dst, double v) { *dst = v; }

__global__ void kc_fill(double *dst, int64_t n, double v) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = v;
}

// transferToGrain (Coupling.cpp:468-527) and then, as nothing between them
// touches the grains, updatePositions_node_node (Coupling.cpp:581-591):
// q = q_before + dt v for every coupled grain (fixed ones are never coupled).
// With hmom the grain, where it then is, adds to the homogenised velocity's
// mass and momentum sums. It is binned there for the next DEM step.
template <int BASIS, bool W32>
__global__ void kc_transfer(const __grid_constant__ GrainArgs A, const __grid_constant__ BinArgs B,
                            const double *a_after, double dt, double *hmom,
                            double *hmass) {
  pdl_wait();
  pdl_trigger();
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b >= A.nb) return;
  if (A.fixed[b]) {
    bin_body(B, b, A.q[3 * b], A.q[3 * b + 1]);
    return;
  }
  const GridGeom &G = A.G;
  double vx = A.v[3 * b], vy = A.v[3 * b + 1], qx, qy;
  GridStencil<BASIS, W32> S;
  if (A.coupled[b]) {
    const double x = A.pos[3 * b], y = A.pos[3 * b + 1], hl = *A.hl0;
    S.range(G, x, y, hl);
    // (the FLIP blend with alpha = 1 leaves v + sum w a_after)
    double ax = 0.0, ay = 0.0;
    visit(S, G, x, y, hl, [&](int64_t i, double wt) {
      const double2 a = reinterpret_cast<const double2 *>(a_after)[i];
      ax = fma(wt, a.x, ax);
      ay = fma(wt, a.y, ay);
    });
    vx += ax;
    vy += ay;
    qx = x + dt * vx;
    qy = y + dt * vy;
    A.v[3 * b] = vx;
    A.v[3 * b + 1] = vy;
    A.q[3 * b] = qx;
    A.q[3 * b + 1] = qy;
  } else {
    qx = A.q[3 * b];
    qy = A.q[3 * b + 1];
  }
  bin_body(B, b, qx, qy);
  if (!hmom) return;
  const double mass = A.m0[b] * A.w[b], hl = G.h * 0.25;
  const double px = mass * vx, py = mass * vy;
  S.range(G, qx, qy, hl);
  visit(S, G, qx, qy, hl, [&](int64_t i, double wt) {
    atomicAdd(&hmom[2 * i], wt * px);
    atomicAdd(&hmom[2 * i + 1], wt * py);
    atomicAdd(&hmass[i], wt * mass);
  });
}

struct HomogenizeArgs {
  GridGeom G;
  int64_t nn;
  int node_blocks; // CTAs over the nodes; the others walk the contacts
  // velocity (nullptr: not homogenised); the sums are cleared here
  double *hmom, *hmass, *hvel;
  // stress (nullptr: not homogenised)
  const int2 *range; // the circle-circle contacts of the contact list
  const double *rec, *q;
  double *hstress;
  double inv_area; // 1 / h^2
};

template <int BASIS, bool W32>
__global__ void __launch_bounds__(128) kc_homogenize(const __grid_constant__ HomogenizeArgs A) {
  pdl_wait();
  pdl_trigger();
  const GridGeom &G = A.G;
  if ((int)blockIdx.x < A.node_blocks) {
    const int64_t i = blockIdx.x * 128ll + threadIdx.x;
    if (i >= A.nn) return;
    const double m = A.hmass[i];
    if (f64_zero(m)) return;
    double2 *hmom = reinterpret_cast<double2 *>(A.hmom), *hvel = reinterpret_cast<double2 *>(A.hvel);
    const double2 p = hmom[i];
    if (m > 0.0) {
      const Divisor M = divisor(m);
      const double2 v = hvel[i];
      hvel[i] = make_double2(v.x + quot(p.x, M), v.y + quot(p.y, M));
    }
    A.hmass[i] = 0.0;
    hmom[i] = make_double2(0.0, 0.0);
    return;
  }
  const int2 r = *A.range;
  const double inv = A.inv_area, hl = G.h * 0.25;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nblocks = (int)gridDim.x - A.node_blocks;
  // chunks of 32 contacts, consecutive ones to different CTAs
  for (int64_t c = blockIdx.x - A.node_blocks + (int64_t)nblocks * wid; r.x + 32 * c < r.y;
       c += 4ll * nblocks) {
    const int64_t k = r.x + 32 * c + lane;
    if (k >= r.y) break;
    const double2 *r_ = reinterpret_cast<const double2 *>(A.rec + k * HG_DEM_RECORD_WIDTH);
    const int b0 = floor_int(r_[0].y), b1 = floor_int(r_[1].x);
    const double px = r_[7].y, py = r_[8].x;
    const double fx = r_[8].y + r_[9].y, fy = r_[9].x + r_[10].x;
    const double rx = A.q[3 * b0] - A.q[3 * b1], ry = A.q[3 * b0 + 1] - A.q[3 * b1 + 1];
    // -0.5 (f r^T + r f^T) / area, column-major (00, 10, 01, 11); symmetric
    const double s00 = -0.5 * (fx * rx + rx * fx) * inv;
    const double s01 = -0.5 * (fx * ry + rx * fy) * inv;
    const double s11 = -0.5 * (fy * ry + ry * fy) * inv;
    GridStencil<BASIS, W32> S;
    S.range(G, px, py, hl);
    visit(S, G, px, py, hl, [&](int64_t i, double wt) {
      const double off = wt * s01;
      atomicAdd(&A.hstress[4 * i], wt * s00);
      atomicAdd(&A.hstress[4 * i + 1], off);
      atomicAdd(&A.hstress[4 * i + 2], off);
      atomicAdd(&A.hstress[4 * i + 3], wt * s11);
    });
  }
}

inline int blocks_for(int64_t n, int t) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }

// the exchange's grids and the homogenisation's sums as before a first step
hg_status clear_grids(hg_hybrid *h) {
  const size_t bytes = sizeof(double) * (size_t)(h->m->p.nx + 1) * (h->m->p.ny + 1);
  for (double *p : {h->dem_mass.p, h->old_mass.p, h->hmass.p})
    HG_CUDA_TRY(cudaMemsetAsync(p, 0, bytes, h->ctx->stream));
  for (double *p : {h->dem_mom.p, h->old_mom.p, h->hmom.p, h->v_after.p, h->a_after.p})
    HG_CUDA_TRY(cudaMemsetAsync(p, 0, 2 * bytes, h->ctx->stream));
  h->grids_kept = true;
  return HG_OK;
}

} // namespace

hg_status hybrid_alloc(hg_hybrid *h) {
  const int64_t nn = (int64_t)(h->m->p.nx + 1) * (h->m->p.ny + 1);
  const int64_t nb = std::max<int64_t>(h->d->cap, 1);
  const int64_t big = std::max(nn, nb) + 1;
  hg_status st;
  if ((st = h->dem_mass.alloc(nn)) || (st = h->dem_mom.alloc(2 * nn)) ||
      (st = h->old_mass.alloc(nn)) || (st = h->old_mom.alloc(2 * nn)) ||
      (st = h->v_after.alloc(2 * nn)) || (st = h->a_after.alloc(2 * nn)) ||
      (st = h->pos_before.alloc(3 * nb)) || (st = h->hstress.alloc(4 * nn)) ||
      (st = h->hvel.alloc(2 * nn)) || (st = h->hmom.alloc(2 * nn)) ||
      (st = h->hmass.alloc(nn)) || (st = h->coupled.alloc(nb + 1)) ||
      (st = h->packed_dem.alloc(nb)) || (st = h->packed_mpm.alloc(nn)) ||
      (st = h->flag_tmp.alloc(big)) || (st = h->scan_tmp.alloc(scan_tmp_size(big))) ||
      (st = h->node_flag.alloc(nn + 1)) || (st = h->node_pos.alloc(nn + 1)) ||
      (st = h->counts.alloc(2)))
    return st;
  cudaStream_t s = h->ctx->stream;
  if (h->m->p.precision == HG_PRECISION_MIXED) {
    if ((st = h->homog.alloc(nn)) || (st = h->hl0.alloc(1))) return st;
    HG_LAUNCH(kc_set_scalar, 1, 1, 0, s, h->hl0.p, 0.0);
    HG_CHECK_LAUNCH();
    h->hl0_value = 0.0;
    HG_LAUNCH(kc_fill, blocks_for(nn, 256), 256, 0, s, h->homog.p, nn, 1.0);
    HG_CHECK_LAUNCH();
  }
  HG_CUDA_TRY(cudaMemsetAsync(h->counts.p, 0, 2 * sizeof(int32_t), s));
  if ((st = clear_grids(h))) return st;
  hg_status r = hybrid_clear_homogenized(h);
  if (r != HG_OK) return r;
  HG_CUDA_TRY(cudaStreamSynchronize(s));
  return HG_OK;
}

hg_status hybrid_pack_lists(hg_hybrid *h) {
  if (h->packed_valid) return HG_OK;
  cudaStream_t s = h->ctx->stream;
  const int64_t nn = (int64_t)(h->m->p.nx + 1) * (h->m->p.ny + 1), nb = h->step_bodies;
  hg_status st;
  // std::stable_partition of the grains (Coupling.cpp:113-127):
  // kc_grain_scatter flagged them
  HG_CUDA_TRY(cudaMemsetAsync(h->coupled.p + nb, 0, sizeof(int32_t), s));
  if ((st = exclusive_scan_i32(h->coupled.p, h->flag_tmp.p, nb + 1, h->scan_tmp.p, s))) return st;
  HG_LAUNCH(kc_pack, blocks_for(nb + 1, 256), 256, 0, s, nb, h->coupled.p, h->flag_tmp.p,
            h->packed_dem.p, h->counts.p);
  HG_CHECK_LAUNCH();
  // and of the nodes with DEM mass
  HG_LAUNCH(kc_flag_nodes, blocks_for(nn, 256), 256, 0, s, nn, h->dem_mass.p, h->node_flag.p);
  HG_CHECK_LAUNCH();
  HG_CUDA_TRY(cudaMemsetAsync(h->node_flag.p + nn, 0, sizeof(int32_t), s));
  if ((st = exclusive_scan_i32(h->node_flag.p, h->node_pos.p, nn + 1, h->scan_tmp.p, s)))
    return st;
  HG_LAUNCH(kc_pack, blocks_for(nn + 1, 256), 256, 0, s, nn, h->node_flag.p, h->node_pos.p,
            h->packed_mpm.p, h->counts.p + 1);
  HG_CHECK_LAUNCH();
  h->packed_valid = true;
  return HG_OK;
}

hg_status hybrid_clear_homogenized(hg_hybrid *h) {
  const int64_t nn = (int64_t)(h->m->p.nx + 1) * (h->m->p.ny + 1);
  cudaStream_t s = h->ctx->stream;
  HG_CUDA_TRY(cudaMemsetAsync(h->hstress.p, 0, sizeof(double) * 4 * nn, s));
  HG_CUDA_TRY(cudaMemsetAsync(h->hvel.p, 0, sizeof(double) * 2 * nn, s));
  return HG_OK;
}

namespace {

// One warp per CTA while the grains are few: a CTA on every SM (9,000 grains:
// 279 CTAs, where CTAs of four warps would leave half of the SMs idle).
int grain_threads(const hg_hybrid *h, int64_t nb) {
  return nb < (int64_t)h->ctx->num_sms * 32 * 16 ? 32 : 128;
}

// W32: the stencil weights of the coupling kernels in FP32 (a MIXED bulk)
template <int BASIS, bool W32> hg_status hybrid_step_impl(hg_hybrid *h, double dt, int flags) {
  using M = std::conditional_t<W32, float, double>; // the MPM node mass type
  hg_mpm *m = h->m;
  hg_dem *d = h->d;
  cudaStream_t s = h->ctx->stream;
  const int64_t nn = (int64_t)(m->p.nx + 1) * (m->p.ny + 1);
  const int64_t nb = d->n;
  hg_status st;
  // (what a failed step scattered, and which set it had taken, is dropped)
  if (!h->grids_kept && (st = clear_grids(h))) return st;
  h->grids_kept = false;
  // A MIXED MPM object (FP32 bulk, FP64 positions) runs the same sequence on
  // its FP32 grid: its P2G for this step was done by the previous particle
  // launch (or the upload), its grid update and G2P are separate launches.
  const double *hl0 = m->hl.p;
  if (W32) {
    if ((st = mixed_step_begin(m))) return st;
    // points.hl(0) in world units: the half-width of the first uploaded point
    const double v = m->p.basis == HG_BASIS_UGIMP ? (double)m->hl_cells * m->p.h : 0.0;
    if (v != h->hl0_value) {
      HG_LAUNCH(kc_set_scalar, 1, 1, 0, s, h->hl0.p, v);
      HG_CHECK_LAUNCH();
      h->hl0_value = v;
    }
    hl0 = h->hl0.p;
  } else {
    // the reference's half gravity of hybridized nodes never applies here: the
    // coupling only clears the flags, which a loaded state alone can set
    if (m->hyb_loaded) HG_CUDA_TRY(cudaMemsetAsync(m->g_hyb.p, 0, sizeof(int32_t) * nn, s));
    m->hyb_loaded = false;
    if ((st = mpm64_to_grid(m))) return st;
  }
  // The coupled grains (flagged by kc_grain_scatter) and nodes (DEM mass > 0)
  // are walked in place: each is handled on its own and the scatters use
  // atomics, so the reference's packed order (Coupling.cpp:113-127) matters
  // only to callers of the lists, which hybrid_pack_lists builds on demand.
  h->packed_valid = false;
  h->step_bodies = nb;
  // the grids of this step's exchange: the set that the last one cleared
  std::swap(h->dem_mass.p, h->old_mass.p);
  std::swap(h->dem_mom.p, h->old_mom.p);
  // DiscreteIntegrator::step -> flowWithWeight (DiscreteIntegrator.cpp:99-116);
  // it keeps the positions before it (copyPrePositionsFull, Coupling.cpp:
  // 529-531), and kc_transfer moves the grains after it
  if ((st = dem_step(d, dt, 1, false, h->pos_before.p))) return st;
  GrainArgs A;
  A.G = geom(m);
  A.nb = nb;
  A.pos = h->pos_before.p;
  A.hl0 = hl0;
  A.fixed = d->fixed.p;
  A.m0 = d->m0.p;
  A.w = d->w.p;
  A.v = d->v.p;
  A.q = d->q.p;
  A.coupled = h->coupled.p;
  const int t = grain_threads(h, nb);
  const M *g_mass;
  if constexpr (W32) g_mass = m->accm.p;
  else g_mass = m->g_mass.p;
  if (nb > 0) {
    auto kernel = kc_grain_scatter<BASIS, W32, M>;
    HG_LAUNCH_PDL(kernel, blocks_for(nb, t), t, 0, s, A, g_mass, h->dem_mass.p, h->dem_mom.p);
    HG_CHECK_LAUNCH();
  }
  if ((st = W32 ? mixed_grid_update(m, dt) : mpm64_phase1(m, dt))) return st;
  // updateVelocitiesOnGrid and the homogenisation factors
  NodeArgs N;
  N.nn = nn;
  N.dem_mass = h->dem_mass.p;
  N.dem_mom = h->dem_mom.p;
  N.old_mass = h->old_mass.p;
  N.old_mom = h->old_mom.p;
  N.v_after = h->v_after.p;
  N.a_after = h->a_after.p;
  N.homog = W32 ? h->homog.p : m->g_homog.p;
  if (W32) {
    HG_LAUNCH_PDL(kc_update_nodes_x, blocks_for(nn, 128), 128, 0, s, N, (const float *)m->gm.p, dt,
                  m->va.p);
  } else {
    HG_LAUNCH_PDL(kc_update_nodes, blocks_for(nn, 128), 128, 0, s, N, (const double *)m->g_mass.p,
                  m->g_mom_new.p);
  }
  HG_CHECK_LAUNCH();
  const bool hv = (flags & HG_HYBRID_HOMOGENIZE_VELOCITY) && nb > 0;
  const bool hs = (flags & HG_HYBRID_HOMOGENIZE_STRESS) && nb > 0;
  if (nb > 0) {
    auto kernel = kc_transfer<BASIS, W32>;
    BinArgs B;
    dem_bin_args(d, &B);
    HG_LAUNCH_PDL(kernel, blocks_for(nb, t), t, 0, s, A, B, (const double *)h->a_after.p, dt,
                  hv ? h->hmom.p : (double *)nullptr, h->hmass.p);
    HG_CHECK_LAUNCH();
    dem_binned(d);
  }
  if ((st = W32 ? mixed_particles(m, dt) : mpm64_phase2(m, dt))) return st;
  if (hv || hs) {
    HomogenizeArgs H;
    H.G = A.G;
    H.nn = nn;
    H.node_blocks = hv ? blocks_for(nn, 128) : 0;
    H.hmom = h->hmom.p;
    H.hmass = h->hmass.p;
    H.hvel = h->hvel.p;
    H.range = d->cc_range.p;
    H.rec = d->crec[d->cc].p;
    H.q = d->q.p;
    H.hstress = h->hstress.p;
    H.inv_area = 1.0 / (m->p.h * m->p.h);
    const int contact_blocks =
        hs ? (int)std::min<int64_t>((d->ccap + 31) / 32, (int64_t)h->ctx->num_sms * 4) : 0;
    auto kernel = kc_homogenize<BASIS, W32>;
    HG_LAUNCH_PDL(kernel, H.node_blocks + contact_blocks, 128, 0, s, H);
    HG_CHECK_LAUNCH();
  }
  h->grids_kept = true;
  return HG_OK;
}

} // namespace

hg_status hybrid_step(hg_hybrid *h, double dt, int flags) {
  const bool mixed = h->m->p.precision == HG_PRECISION_MIXED;
  if (h->m->p.basis == HG_BASIS_UGIMP)
    return mixed ? hybrid_step_impl<HG_BASIS_UGIMP, true>(h, dt, flags)
                 : hybrid_step_impl<HG_BASIS_UGIMP, false>(h, dt, flags);
  return mixed ? hybrid_step_impl<HG_BASIS_LINEAR, true>(h, dt, flags)
               : hybrid_step_impl<HG_BASIS_LINEAR, false>(h, dt, flags);
}

} // namespace hg
