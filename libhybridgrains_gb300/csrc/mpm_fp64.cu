// Plain FP64 MPM step: the drop-in for ExplicitIntegrator::flow in double
// precision.
//
// Bound by the FP64 pipe: an FP64 instruction takes a warp 64 cycles whatever
// it does (fp64_tools.cuh), so each kernel evaluates what the reference
// evaluates in as few FP64 instructions as keep its accuracy. Positions, cells,
// stencil offsets, strains and plane tests, where a last bit decides or
// survives a cancellation, keep the reference's operations one by one (this
// translation unit is compiled with --fmad=false); sums and products elsewhere
// use fma() explicitly, quotients by a common divisor share its reciprocal,
// roots come with theirs, 1-D factors are divided once per axis, and sign,
// range and yield decisions are made on the integer and FP32 pipes with an FP64
// test for the close calls. Grid accumulation uses FP64 atomics, so node sums
// differ from the serial reference in order too; both stay within a few units
// in the last place (tests: 1e-12).
// Measured per step against the reference's expressions instruction for
// instruction (six memsets and four launches a step, now three launches):
// 12,800 points, linear, one call per step 84.5 -> 22.4 us; 100,000 points,
// uGIMP, 439 -> 118 us (k64_g2p 214 -> 65 us: 286 FP64 instructions per warp
// of points where there were about 1,100, 81% of the FP64 pipe; k64_p2g 170 ->
// 50 us).
//
// Kernels:
//   k64_p2g         rasterizePointMasses + rasterizePointMomentum
//                   (PhysicsGrid.cpp:168-411), computeHyperelasticCauchyStress
//                   (MaterialPoints.cpp:183-202) and the particle part of
//                   computeForces (PhysicsGrid.cpp:413-471)
//   k64_grid        node part of computeForces (PhysicsGrid.cpp:459-471),
//                   updateMomentum (565-586), resolvePlaneCollisions
//                   (611-673) and lumpedMassVelocityAndAccelerationUpdate
//                   (588-609); as two launches where a caller acts in between
//   k64_g2p         computeVelGrad, elasticPrediction, plasticCorrection,
//                   updateVelocities, updatePositions, resolvePlaneCollisions
//                   (MaterialPoints.cpp:204-423), fused per material point;
//                   clears the accumulators of the next step.
#include "hg_internal.cuh"
#include "mpm_basis.cuh"
#include "mpm_axis.cuh"

#include <cmath>
#include <utility>

namespace hg {

namespace {

struct M2d {
  double a00, a10, a01, a11;
};

__device__ __forceinline__ M2d m_add(M2d a, M2d b) {
  return {a.a00 + b.a00, a.a10 + b.a10, a.a01 + b.a01, a.a11 + b.a11};
}
__device__ __forceinline__ M2d m_sub(M2d a, M2d b) {
  return {a.a00 - b.a00, a.a10 - b.a10, a.a01 - b.a01, a.a11 - b.a11};
}
__device__ __forceinline__ M2d m_scl(double s, M2d a) {
  return {s * a.a00, s * a.a10, s * a.a01, s * a.a11};
}
__device__ __forceinline__ M2d m_div(M2d a, double s) {
  return {a.a00 / s, a.a10 / s, a.a01 / s, a.a11 / s};
}
__device__ __forceinline__ M2d m_mul(M2d a, M2d b) {
  return {a.a00 * b.a00 + a.a01 * b.a10, a.a10 * b.a00 + a.a11 * b.a10,
          a.a00 * b.a01 + a.a01 * b.a11, a.a10 * b.a01 + a.a11 * b.a11};
}
__device__ __forceinline__ M2d m_T(M2d a) { return {a.a00, a.a01, a.a10, a.a11}; }
__device__ __forceinline__ double m_det(M2d a) {
  return a.a00 * a.a11 - a.a10 * a.a01;
}
__device__ __forceinline__ double m_tr(M2d a) { return a.a00 + a.a11; }
__device__ __forceinline__ double m_norm(M2d a) {
  return sqrt(a.a00 * a.a00 + a.a10 * a.a10 + a.a01 * a.a01 + a.a11 * a.a11);
}
__device__ __forceinline__ M2d m_id(double s) { return {s, 0.0, 0.0, s}; }

// ConstitutiveModel.cpp:26-81
__device__ M2d plastic_correction(M2d b, double kappa, double mu, double alpha,
                                  int &jh) {
  if (jh != 0) {
    const double J = sqrt(m_det(b));
    if (J > 1.0) return m_id(J);
    jh = 0;
  }
  const double J = sqrt(m_det(b));
  const double ys = fmax(0.0, 0.5 * alpha * kappa * (1.0 + J) * (1.0 - J));
  const double half_tr = 0.5 * m_tr(b);
  const M2d dev = m_sub(b, m_id(half_tr));
  const M2d bar_dev = m_div(dev, J);
  if (mu * m_norm(bar_dev) > ys) {
    const double lambda2 = ys / (mu * m_norm(bar_dev));
    const double l1sq = m_det(b) - lambda2 * lambda2 * m_det(dev);
    const double lambda1 = sqrt(l1sq);
    return m_add(m_id(lambda1), m_scl(lambda2, dev));
  }
  return b;
}

// A point's stencil: the 2-D weight of node (kx, ky) is wx[kx] wy[ky] and its
// gradient (dx[kx] wy[ky], wx[kx] dy[ky]).
template <int BASIS> struct Stencil;
template <> struct Stencil<HG_BASIS_LINEAR> {
  using Ax = Axis<HG_BASIS_LINEAR>;
  Ax X, Y;
  template <bool SAFE>
  __device__ __forceinline__ void set(const MpmParams &P, double x, double y, double hl,
                                      const Divisor &H, bool &ok) {
    X.template range<SAFE>(x, hl, P.gmin[0], H, ok);
    Y.template range<SAFE>(y, hl, P.gmin[1], H, ok);
    X.template factors<true, SAFE>(x, P.gmin[0], H, ok);
    Y.template factors<true, SAFE>(y, P.gmin[1], H, ok);
  }
  template <class F> __device__ __forceinline__ void each(int row, F &&f) const {
#pragma unroll
    for (int ky = 0; ky < 2; ++ky)
#pragma unroll
      for (int kx = 0; kx < 2; ++kx)
        f((Y.i0 + ky) * (int64_t)row + X.i0 + kx, X.w[kx] * Y.w[ky],
          X.sg[kx] == Ax::NO_SLOPE ? 0.0 : flip(Y.v[ky], X.sg[kx]),
          Y.sg[ky] == Ax::NO_SLOPE ? 0.0 : flip(X.v[kx], Y.sg[ky]));
  }
};
template <> struct Stencil<HG_BASIS_UGIMP> {
  Axis<HG_BASIS_UGIMP> X, Y;
  template <bool SAFE>
  __device__ __forceinline__ void set(const MpmParams &P, double x, double y, double hl,
                                      const Divisor &H, bool &ok) {
    Extent E;
    E.set(hl, H);
    X.template range<SAFE>(x, hl, P.gmin[0], H, ok);
    Y.template range<SAFE>(y, hl, P.gmin[1], H, ok);
    X.factors<true>(x, E, P.gmin[0], H);
    Y.factors<true>(y, E, P.gmin[1], H);
    // over the point's volume 4 hl^2, once per node of one axis
    const double inv = 1.0 / (4.0 * hl * hl);
#pragma unroll
    for (int k = 0; k < STENCIL_AXIS; ++k)
      if (k < Y.n) {
        Y.w[k] *= inv;
        Y.d[k] *= inv;
      }
  }
};

template <int BASIS>
__device__ __noinline__ Stencil<BASIS> stencil_safe(const MpmParams &P, double x, double y,
                                                    double hl) {
  Stencil<BASIS> S;
  bool ok = true;
  S.template set<true>(P, x, y, hl, divisor(P.h, P.inv_h), ok);
  return S;
}
template <int BASIS>
__device__ __forceinline__ void stencil(Stencil<BASIS> &S, const MpmParams &P, double x, double y,
                                        double hl) {
  const Divisor H = divisor(P.h, P.inv_h);
  bool ok = H.ok;
  S.template set<false>(P, x, y, hl, H, ok);
  if (!ok) S = stencil_safe<BASIS>(P, x, y, hl);
}

// The node range leaves the grid, or is wider than the kernels' stencils hold.
template <int BASIS>
__device__ __forceinline__ bool off_grid(const MpmParams &P, const Stencil<BASIS> &S) {
  return S.X.i0 < 0 || S.Y.i0 < 0 || S.X.i0 + S.X.n - 1 > P.nx || S.Y.i0 + S.Y.n - 1 > P.ny;
}
template <int BASIS> __device__ __forceinline__ bool too_wide(const Stencil<BASIS> &S) {
  return BASIS == HG_BASIS_UGIMP && (S.X.n > STENCIL_AXIS || S.Y.n > STENCIL_AXIS);
}

struct P2gArgs {
  int64_t n;
  const double *q, *v, *m, *vol, *hl, *be, *J;
  const int32_t *jh;
  double *g_mass, *g_mom, *g_force;
  uint32_t *status;
  double half_kappa;
};

// Strains are stored as be_bar and J near 1, so the last bit of each is the
// last bit of the stress: what forms them (products with J, determinants,
// roots, quotients, traces) keeps the reference's operations one by one.
__device__ __forceinline__ double det_sym(double b00, double b01, double b11) {
  return b00 * b11 - b01 * b01;
}

// -vol tau, the Kirchhoff stress as it enters the node forces
// (-vol J sigma with sigma = tau / J), ConstitutiveModel.cpp:83-97.
__device__ __forceinline__ M2d node_stress(const MpmParams &P, const P2gArgs &A, int64_t p) {
  const double Jp = A.J[p];
  if (!(Jp <= 1.0) || A.jh[p] != 0) {
    // (no stress is 0 / J: a J that is not a number reaches the nodes)
    const double none = finite_bits(Jp) && !f64_zero(Jp) ? 0.0 : __hiloint2double(0x7FF80000, 0);
    return {none, none, none, none};
  }
  const double2 c0 = reinterpret_cast<const double2 *>(A.be)[2 * p];
  const double2 c1 = reinterpret_cast<const double2 *>(A.be)[2 * p + 1];
  const M2d be = m_scl(Jp, M2d{c0.x, c0.y, c1.x, c1.y});
  const double2 r = root(m_det(be));
  const double J = r.x;
  const Divisor D = divisor(J, r.y);
  bool ok = D.ok;
  double a00 = quot(be.a00, D, ok), a10 = quot(be.a10, D, ok), a11 = quot(be.a11, D, ok);
  double a01 = a10;
  if (__double_as_longlong(c0.y) != __double_as_longlong(c1.x)) a01 = quot(be.a01, D, ok);
  if (!ok) {
    a00 = divide(be.a00, J);
    a10 = divide(be.a10, J);
    a01 = divide(be.a01, J);
    a11 = divide(be.a11, J);
  }
  const double half_tr = halved(a00 + a11);
  const double s = A.half_kappa * (J + 1.0) * (J - 1.0);
  const double c = -A.vol[p], cm = c * P.mu;
  return {c * fma(P.mu, a00 - half_tr, s), cm * a10, cm * a01, c * fma(P.mu, a11 - half_tr, s)};
}

// General stencils (wider than STENCIL_AXIS nodes), node by node.
__device__ __noinline__ void p2g_wide(const MpmParams &P, const P2gArgs &A, int64_t p, M2d S) {
  const double x = A.q[2 * p], y = A.q[2 * p + 1], h = A.hl[p], mp = A.m[p];
  const double pmx = mp * A.v[2 * p], pmy = mp * A.v[2 * p + 1];
  int x0, y0, x1, y1;
  stencil64(P.basis, x, y, h, P.gmin[0], P.gmin[1], P.h, x0, y0, x1, y1);
  for (int iy = y0; iy <= y1; ++iy)
    for (int ix = x0; ix <= x1; ++ix) {
      double gx, gy;
      weight_grad64(P.basis, x, y, h, ix, iy, P.gmin[0], P.gmin[1], P.h, gx, gy);
      const double w = weight64(P.basis, x, y, h, ix, iy, P.gmin[0], P.gmin[1], P.h);
      const int64_t i = (int64_t)iy * (P.nx + 1) + ix;
      atomicAdd(&A.g_mass[i], w * mp);
      atomicAdd(&A.g_mom[2 * i], w * pmx);
      atomicAdd(&A.g_mom[2 * i + 1], w * pmy);
      if (w == 0.0) continue;
      atomicAdd(&A.g_force[2 * i], S.a00 * gx + S.a01 * gy);
      atomicAdd(&A.g_force[2 * i + 1], S.a10 * gx + S.a11 * gy);
    }
}

template <int BASIS>
__global__ void k64_p2g(const __grid_constant__ MpmParams P, const __grid_constant__ P2gArgs A) {
  pdl_wait();
  pdl_trigger();
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= A.n) return;
  const double2 x = reinterpret_cast<const double2 *>(A.q)[p];
  Stencil<BASIS> St;
  stencil(St, P, x.x, x.y, BASIS == HG_BASIS_UGIMP ? A.hl[p] : 0.0);
  if (off_grid<BASIS>(P, St)) {
    atomicOr(A.status, (uint32_t)HG_STATUS_OUT_OF_GRID);
    return;
  }
  const M2d S = node_stress(P, A, p);
  if (too_wide<BASIS>(St)) {
    p2g_wide(P, A, p, S);
    return;
  }
  const double mp = A.m[p];
  const double2 v = reinterpret_cast<const double2 *>(A.v)[p];
  const double pmx = mp * v.x, pmy = mp * v.y;
  const int row = P.nx + 1;
  // (nodes of zero weight get nothing, PhysicsGrid.cpp:439-441)
  if constexpr (BASIS == HG_BASIS_LINEAR) {
    St.each(row, [&](int64_t i, double w, double gx, double gy) {
      if (f64_zero(w)) return;
      atomicAdd(&A.g_mass[i], w * mp);
      atomicAdd(&A.g_mom[2 * i], w * pmx);
      atomicAdd(&A.g_mom[2 * i + 1], w * pmy);
      atomicAdd(&A.g_force[2 * i], fma(S.a00, gx, S.a01 * gy));
      atomicAdd(&A.g_force[2 * i + 1], fma(S.a10, gx, S.a11 * gy));
    });
  } else {
    // the factors of a row of nodes once per row
#pragma unroll
    for (int ky = 0; ky < STENCIL_AXIS; ++ky) {
      if (ky >= St.Y.n) break;
      const double wy = St.Y.w[ky], dy = St.Y.d[ky];
      if (f64_zero(wy)) continue;
      const double rm = wy * mp, rx = wy * pmx, ry = wy * pmy;
      const double f00 = S.a00 * wy, f10 = S.a10 * wy, f01 = S.a01 * dy, f11 = S.a11 * dy;
      const int64_t base = (St.Y.i0 + ky) * (int64_t)row + St.X.i0;
#pragma unroll
      for (int kx = 0; kx < STENCIL_AXIS; ++kx) {
        if (kx >= St.X.n) break;
        const double wx = St.X.w[kx], dx = St.X.d[kx];
        if (f64_zero(wx)) continue;
        const int64_t i = base + kx;
        atomicAdd(&A.g_mass[i], wx * rm);
        atomicAdd(&A.g_mom[2 * i], wx * rx);
        atomicAdd(&A.g_mom[2 * i + 1], wx * ry);
        atomicAdd(&A.g_force[2 * i], fma(dx, f00, wx * f01));
        atomicAdd(&A.g_force[2 * i + 1], fma(dx, f10, wx * f11));
      }
    }
  }
}

struct GridArgs {
  int64_t nn;
  double dt, inv_dt;
  const double *mass, *mom;
  double *mom_new, *force;
  const double *cforce;
  const int32_t *hyb;
  double *vel, *acc;
  // cells about each plane and its lower bound within which FP64 decides
  float margin[HG_MAX_PLANES], bound_margin[HG_MAX_PLANES];
};

// True when the plane acts on node (ix, iy) (PhysicsGrid.cpp:614-629): in FP32
// grid units away from the plane and its lower bound, within margin and
// bound_margin cells of them by the reference's own FP64 test.
__device__ __forceinline__ bool node_hit(const MpmParams &P, const MpmPlaneDev &pl, float margin,
                                         float bound_margin, int ix, int iy) {
  const float fx = (float)ix, fy = (float)iy;
  if (fy < pl.fulb - bound_margin) return false;
  const float d32 = pl.fn[0] * (fx - pl.fux[0]) + pl.fn[1] * (fy - pl.fux[1]);
  if (fabsf(d32) > margin && fabsf(fy - pl.fulb) > bound_margin) return d32 < 0.0f;
  const double px = P.gmin[0] + P.h * (double)ix, py = P.gmin[1] + P.h * (double)iy;
  if (py < pl.lower_bound) return false;
  return !(pl.n[0] * (px - pl.x[0]) + pl.n[1] * (py - pl.x[1]) > 0.0);
}

// FORCES: the node forces and new momenta; UPDATE: velocities and
// accelerations from them. Nodes without mass take no FP64 arithmetic.
template <bool FORCES, bool UPDATE>
__global__ void __launch_bounds__(128) k64_grid(const __grid_constant__ MpmParams P,
                                                const __grid_constant__ GridArgs A) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.nn) return;
  double2 *mom_new = reinterpret_cast<double2 *>(A.mom_new);
  const double mi = A.mass[i];
  const bool has = mi > 0.0;
  const double2 zero = make_double2(0.0, 0.0);
  double2 pn = zero, pm = zero;
  if (has) pm = reinterpret_cast<const double2 *>(A.mom)[i];
  if (FORCES) {
    double2 *force = reinterpret_cast<double2 *>(A.force);
    const double2 cf = reinterpret_cast<const double2 *>(A.cforce)[i];
    if (has) {
      double2 f = force[i];
      const double half = A.hyb[i] > 0 ? 0.5 * mi : mi;
      f.x = fma(half, P.g[0], f.x);
      f.y = fma(half, P.g[1], f.y);
      if (!f64_zero(cf.x)) f.x += cf.x;
      if (!f64_zero(cf.y)) f.y += cf.y;
      force[i] = f;
      pn = make_double2(fma(A.dt, f.x, pm.x), fma(A.dt, f.y, pm.y));
      const int ix = (int)(i % (P.nx + 1)), iy = (int)(i / (P.nx + 1));
      for (int k = 0; k < P.nplanes; ++k) { // PhysicsGrid::resolvePlaneCollisions
        const MpmPlaneDev &pl = P.planes[k];
        if (!node_hit(P, pl, A.margin[k], A.bound_margin[k], ix, iy)) continue;
        if (!pl.sticking) {
          double vx = pn.x / mi, vy = pn.y / mi;
          const double vn = pl.n[0] * vx + pl.n[1] * vy;
          if (vn > 0.0) continue;
          vx = vx - vn * pl.n[0];
          vy = vy - vn * pl.n[1];
          pn = make_double2(mi * vx, mi * vy);
        } else {
          pn = zero;
        }
      }
    } else if (!f64_zero(cf.x) || !f64_zero(cf.y)) {
      const double2 f = force[i];
      force[i] = make_double2(f.x + cf.x, f.y + cf.y);
    }
    mom_new[i] = pn;
  } else if (has) {
    pn = mom_new[i];
  }
  if (UPDATE) {
    double2 v = zero, a = zero;
    if (has) {
      const Divisor M = divisor(mi);
      const double per = M.y * A.inv_dt;
      v = make_double2(quot(pn.x, M), quot(pn.y, M));
      a = make_double2((pn.x - pm.x) * per, (pn.y - pm.y) * per);
    }
    reinterpret_cast<double2 *>(A.vel)[i] = v;
    reinterpret_cast<double2 *>(A.acc)[i] = a;
  }
}

struct G2pArgs {
  int64_t n, nn;
  double dt;
  double *q, *v;
  const double *hl;
  double *be, *J;
  int32_t *jh;
  const uint8_t *kin;
  const double *g_vel, *g_acc;
  double *next_mass, *next_mom, *next_force; // the next step's accumulators, cleared
  uint32_t *status;
  // constants of every point
  double yield_mu; // alpha kappa / (2 mu); NaN without a shear modulus
  double pic;   // 1 - flip_alpha
  float mu32, yield32;
  float px[HG_MAX_PLANES][2];
};

// What the grid gives a point: its velocity gradient, velocity, acceleration.
struct PointGrid {
  double L00, L10, L01, L11, vx, vy, ax, ay;
};

__device__ __noinline__ PointGrid g2p_wide(const MpmParams &P, const G2pArgs &A, double x, double y,
                                           double h) {
  PointGrid g{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int x0, y0, x1, y1;
  stencil64(P.basis, x, y, h, P.gmin[0], P.gmin[1], P.h, x0, y0, x1, y1);
  for (int iy = y0; iy <= y1; ++iy)
    for (int ix = x0; ix <= x1; ++ix) {
      double gx, gy;
      weight_grad64(P.basis, x, y, h, ix, iy, P.gmin[0], P.gmin[1], P.h, gx, gy);
      const double w = weight64(P.basis, x, y, h, ix, iy, P.gmin[0], P.gmin[1], P.h);
      const int64_t i = (int64_t)iy * (P.nx + 1) + ix;
      const double vx = A.g_vel[2 * i], vy = A.g_vel[2 * i + 1];
      g.L00 += vx * gx;
      g.L10 += vy * gx;
      g.L01 += vx * gy;
      g.L11 += vy * gy;
      g.vx += w * vx;
      g.vy += w * vy;
      g.ax += w * A.g_acc[2 * i];
      g.ay += w * A.g_acc[2 * i + 1];
    }
  return g;
}

// elasticPrediction and plasticCorrection of a be_bar that is not symmetric
// (MaterialPoints.cpp:324-369, ConstitutiveModel.cpp:19-81), component by
// component.
struct PointStrain {
  M2d b;
  double J;
  int jh;
};
__device__ __noinline__ PointStrain strain_general(const MpmParams &P, double dt, const PointGrid &g,
                                                   PointStrain s) {
  const M2d L{g.L00, g.L10, g.L01, g.L11};
  const M2d ben = m_scl(s.J, s.b);
  const M2d bs = m_add(ben, m_scl(dt, m_add(m_mul(L, ben), m_mul(ben, m_T(L)))));
  const double J1 = sqrt(m_det(bs));
  int jh = s.jh;
  const M2d bn = plastic_correction(m_scl(J1, m_div(bs, J1)), P.kappa, P.mu, P.dp_alpha, jh);
  const double J2 = sqrt(m_det(bn));
  return {m_div(bn, J2), J2, jh};
}

// The same for a symmetric be_bar, which stays symmetric to the bit. The
// yield test is decided in FP32 except within 1e-5 of the yield surface, so
// that elastic points need neither |dev be| nor the yield stress in FP64.
// False when a quotient did not pass its check.
__device__ __forceinline__ bool strain_symmetric(const MpmParams &P, const G2pArgs &A,
                                                 const PointGrid &g, PointStrain &s) {
  bool ok = true;
  double b00 = s.J * s.b.a00, b01 = s.J * s.b.a01, b11 = s.J * s.b.a11;
  const double l00 = fma(g.L00, b00, g.L01 * b01), l01 = fma(g.L00, b01, g.L01 * b11);
  const double l10 = fma(g.L10, b00, g.L11 * b01), l11 = fma(g.L10, b01, g.L11 * b11);
  b00 = fma(A.dt, twice(l00), b00);
  b01 = fma(A.dt, l01 + l10, b01);
  b11 = fma(A.dt, twice(l11), b11);
  {
    const double2 r = root(det_sym(b00, b01, b11));
    const Divisor D = divisor(r.x, r.y);
    ok = D.ok;
    b00 = r.x * quot(b00, D, ok);
    b01 = r.x * quot(b01, D, ok);
    b11 = r.x * quot(b11, D, ok);
  }
  const double det = det_sym(b00, b01, b11);
  double2 r = root(det); // J and 1 / J
  double J = r.x;
  int jh = s.jh;
  const bool grown = jh != 0 && J > 1.0;
  if (!grown) jh = 0;
  if (grown) { // be = J I (ConstitutiveModel.cpp:28-35)
    b00 = b11 = J;
    b01 = 0.0;
    r = root(J * J);
  } else {
    const double half_tr = halved(b00 + b11);
    const double d0 = b00 - half_tr, d1 = b11 - half_tr;
    const double up = 1.0 + J, down = 1.0 - J;
    const float d32 = narrow_trunc(d0), o32 = narrow_trunc(b01);
    const float n2 = 2.0f * (d32 * d32 + o32 * o32);
    const float limit =
        fmaxf(0.0f, A.yield32 * narrow_trunc(up) * narrow_trunc(down)) * narrow_trunc(J) / A.mu32;
    // elastic for sure, where the estimate of |dev be| is well above the
    // rounding of d0 and FP32's smallest squares
    const bool elastic = n2 > 1.0e-18f && sqrtf(n2) < limit * 0.99999f;
    if (!elastic) {
      // l2 = ys / (mu |dev be| / J), below 1 beyond the yield surface; no
      // deviator gives infinity or NaN, no shear modulus NaN (arithmetic's, whose
      // sign bit is clear): neither is below 1
      const double o2 = b01 * b01;
      double l2 = A.yield_mu * up * down * J * rsqrt(fma(d0, d0, fma(d1, d1, twice(o2))));
      if (f64_hi(l2) >> 31) l2 = 0.0; // J > 1: no yield stress
      if (l2 < 1.0) {
        const double l1 = root(fma(-(l2 * l2), fma(d0, d1, -o2), det)).x;
        b00 = fma(l2, d0, l1);
        b11 = fma(l2, d1, l1);
        b01 = l2 * b01;
        r = root(det_sym(b00, b01, b11));
      }
    }
  }
  J = r.x;
  const Divisor D = divisor(J, r.y);
  ok = ok && D.ok;
  const double a00 = quot(b00, D, ok), a01 = quot(b01, D, ok), a11 = quot(b11, D, ok);
  if (ok) s = {{a00, a01, a01, a11}, J, jh};
  return ok;
}

template <int BASIS>
__global__ void k64_g2p(const __grid_constant__ MpmParams P, const __grid_constant__ G2pArgs A) {
  pdl_wait();
  pdl_trigger();
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t i = p; i < A.nn; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 zero = make_double2(0.0, 0.0);
    A.next_mass[i] = 0.0;
    reinterpret_cast<double2 *>(A.next_mom)[i] = zero;
    reinterpret_cast<double2 *>(A.next_force)[i] = zero;
  }
  if (p >= A.n) return;
  double2 x = reinterpret_cast<const double2 *>(A.q)[p];
  const double hl = BASIS == HG_BASIS_UGIMP ? A.hl[p] : 0.0;
  PointGrid g{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  {
    Stencil<BASIS> St;
    stencil(St, P, x.x, x.y, hl);
    if (off_grid<BASIS>(P, St)) {
      atomicOr(A.status, (uint32_t)HG_STATUS_OUT_OF_GRID);
      return;
    }
    if (too_wide<BASIS>(St)) {
      g = g2p_wide(P, A, x.x, x.y, hl);
    } else {
      // computeVelGrad (MaterialPoints.cpp:296-322), and the interpolations of
      // updateVelocities (204-245) and updatePositions (247-288)
      const double2 *gv = reinterpret_cast<const double2 *>(A.g_vel);
      const double2 *ga = reinterpret_cast<const double2 *>(A.g_acc);
      const int row = P.nx + 1;
      if constexpr (BASIS == HG_BASIS_LINEAR) {
        St.each(row, [&](int64_t i, double w, double gx, double gy) {
          const double2 v = gv[i], a = ga[i];
          g.L00 = fma(v.x, gx, g.L00);
          g.L10 = fma(v.y, gx, g.L10);
          g.L01 = fma(v.x, gy, g.L01);
          g.L11 = fma(v.y, gy, g.L11);
          g.vx = fma(w, v.x, g.vx);
          g.vy = fma(w, v.y, g.vy);
          g.ax = fma(w, a.x, g.ax);
          g.ay = fma(w, a.y, g.ay);
        });
      } else {
        // row by row: the sums over x, then their factors along y
#pragma unroll
        for (int ky = 0; ky < STENCIL_AXIS; ++ky) {
          if (ky >= St.Y.n) break;
          const int64_t base = (St.Y.i0 + ky) * (int64_t)row + St.X.i0;
          double vx = 0.0, vy = 0.0, dvx = 0.0, dvy = 0.0, ax = 0.0, ay = 0.0;
#pragma unroll
          for (int kx = 0; kx < STENCIL_AXIS; ++kx) {
            if (kx >= St.X.n) break;
            const double2 v = gv[base + kx], a = ga[base + kx];
            const double w = St.X.w[kx], d = St.X.d[kx];
            vx = fma(w, v.x, vx);
            vy = fma(w, v.y, vy);
            dvx = fma(d, v.x, dvx);
            dvy = fma(d, v.y, dvy);
            ax = fma(w, a.x, ax);
            ay = fma(w, a.y, ay);
          }
          const double wy = St.Y.w[ky], dy = St.Y.d[ky];
          g.L00 = fma(wy, dvx, g.L00);
          g.L10 = fma(wy, dvy, g.L10);
          g.L01 = fma(dy, vx, g.L01);
          g.L11 = fma(dy, vy, g.L11);
          g.vx = fma(wy, vx, g.vx);
          g.vy = fma(wy, vy, g.vy);
          g.ax = fma(wy, ax, g.ax);
          g.ay = fma(wy, ay, g.ay);
        }
      }
    }
  }
  PointStrain s;
  {
    const double2 c0 = reinterpret_cast<const double2 *>(A.be)[2 * p];
    const double2 c1 = reinterpret_cast<const double2 *>(A.be)[2 * p + 1];
    s = {{c0.x, c0.y, c1.x, c1.y}, A.J[p], A.jh[p]};
  }
  if (__double_as_longlong(s.b.a10) != __double_as_longlong(s.b.a01) ||
      !strain_symmetric(P, A, g, s))
    s = strain_general(P, A.dt, g, s);
  double2 v = reinterpret_cast<const double2 *>(A.v)[p];
  if (A.kin[p] == 0) {
    const double a = P.flip_alpha, b = A.pic;
    v.x = fma(a, fma(g.ax, A.dt, v.x), b * g.vx);
    v.y = fma(a, fma(g.ay, A.dt, v.y), b * g.vy);
    x.x += A.dt * g.vx;
    x.y += A.dt * g.vy;
  } else {
    x.x += A.dt * v.x;
    x.y += A.dt * v.y;
  }
  // MaterialPoints::resolvePlaneCollisions (MaterialPoints.cpp:371-423): FP32
  // leaves out the planes a point is clearly in front of (the coordinates'
  // truncation and FP32 sums err by less than 1e-6 of the terms)
  for (int k = 0; k < P.nplanes; ++k) {
    const MpmPlaneDev &pl = P.planes[k];
    {
      const float fx = narrow_trunc(x.x), fy = narrow_trunc(x.y);
      const float px = A.px[k][0], py = A.px[k][1];
      const float d32 = pl.fn[0] * (fx - px) + pl.fn[1] * (fy - py);
      if (d32 > 1.0e-6f * (fabsf(fx) + fabsf(px) + fabsf(fy) + fabsf(py))) continue;
    }
    if (x.y < pl.lower_bound) continue;
    const double d = pl.n[0] * (x.x - pl.x[0]) + pl.n[1] * (x.y - pl.x[1]);
    if (d > 0.0) continue;
    x.x += -d * pl.n[0];
    x.y += -d * pl.n[1];
    if (!pl.sticking) {
      const double vn = pl.n[0] * v.x + pl.n[1] * v.y;
      if (vn > 0.0) continue;
      v.x = v.x - vn * pl.n[0];
      v.y = v.y - vn * pl.n[1];
    } else {
      v = make_double2(0.0, 0.0);
    }
  }
  if (!finite_bits(x.x) || !finite_bits(x.y) || !finite_bits(v.x) || !finite_bits(v.y) ||
      !finite_bits(s.J))
    atomicOr(A.status, (uint32_t)HG_STATUS_NONFINITE);
  reinterpret_cast<double2 *>(A.q)[p] = x;
  reinterpret_cast<double2 *>(A.v)[p] = v;
  reinterpret_cast<double2 *>(A.be)[2 * p] = make_double2(s.b.a00, s.b.a10);
  reinterpret_cast<double2 *>(A.be)[2 * p + 1] = make_double2(s.b.a01, s.b.a11);
  A.J[p] = s.J;
  A.jh[p] = s.jh;
}

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

// Threads per CTA of the point kernels: one warp while the points are few, so
// that their warps spread over all SMs' FP64 pipes (12,800 points: 400 warps,
// at most 3 per SM against 4 with CTAs of four warps).
int point_threads(const hg_mpm *m) {
  return m->n < (int64_t)m->ctx->num_sms * 32 * 16 ? 32 : 128;
}

// CTAs of the kernel that moves the points and clears the next accumulators: one
// thread per point, more where a thread would clear more than eight nodes, up to
// a chip full. (With the points' alone a point on a grid of 1000 x 1000 cells took
// 634 us per step, now 32; 300 points on 3000 x 3000 cells 2,260 and 160.)
int g2p_blocks(const hg_mpm *m, int64_t nodes, int t) {
  const int clearing = (int)std::min<int64_t>(blocks_for(nodes, 8 * t), m->ctx->num_sms * 1024 / t);
  return std::max(blocks_for(m->n, t), clearing);
}

template <bool FORCES, bool UPDATE> hg_status grid_pass(hg_mpm *m, double dt) {
  GridArgs A;
  A.nn = (int64_t)(m->p.nx + 1) * (m->p.ny + 1);
  A.dt = dt;
  A.inv_dt = 1.0 / dt;
  A.mass = m->g_mass.p;
  A.mom = m->g_mom.p;
  A.mom_new = m->g_mom_new.p;
  A.force = m->g_force.p;
  A.cforce = m->g_cforce.p;
  A.hyb = m->g_hyb.p;
  A.vel = m->g_vel.p;
  A.acc = m->g_acc.p;
  // A normal's component, an anchor's coordinate, their difference, product and
  // sum each round by 2^-24 of a term, the terms being at most the grid's extent
  // and the anchor's distance: five of them are 3e-7 of the terms. (The FP64 test
  // itself rounds at the grid's distance from the origin: well below 0.01 cells
  // of any grid whose nodes are distinct numbers by that much.)
  for (int k = 0; k < m->p.nplanes; ++k) {
    const MpmPlaneDev &pl = m->p.planes[k];
    const double size = (double)m->p.nx + m->p.ny;
    A.margin[k] = (float)(0.01 + 4.0e-7 * (size + std::fabs(pl.ux[0]) + std::fabs(pl.ux[1])));
    A.bound_margin[k] =
        std::isfinite(pl.ulb) ? (float)(0.01 + 4.0e-7 * (size + std::fabs(pl.ulb))) : 0.01f;
  }
  auto kernel = k64_grid<FORCES, UPDATE>;
  HG_LAUNCH_PDL(kernel, blocks_for(A.nn, 128), 128, 0, m->ctx->stream, m->p, A);
  HG_CHECK_LAUNCH();
  return HG_OK;
}

hg_status to_points(hg_mpm *m, double dt) {
  if (m->n <= 0) return HG_OK;
  G2pArgs A;
  A.n = m->n;
  A.nn = (int64_t)(m->p.nx + 1) * (m->p.ny + 1);
  A.dt = dt;
  A.q = m->q.p;
  A.v = m->v.p;
  A.hl = m->hl.p;
  A.be = m->be.p;
  A.J = m->J.p;
  A.jh = m->jh.p;
  A.kin = m->kin.p;
  A.g_vel = m->g_vel.p;
  A.g_acc = m->g_acc.p;
  A.next_mass = m->g_mass_next.p;
  A.next_mom = m->g_mom_next.p;
  A.next_force = m->g_force_next.p;
  A.status = m->status.p;
  const double yield = 0.5 * m->p.dp_alpha * m->p.kappa;
  // (without a shear modulus mu |dev be| exceeds no yield stress; a test of its
  // own on the device cost 12,800 to 52,000 points 7 to 28 % of the step, through
  // the registers and so the places of the next kernel's CTAs)
  A.yield_mu = m->p.mu > 0.0 ? yield / m->p.mu : std::nan("");
  A.pic = 1.0 - m->p.flip_alpha;
  A.mu32 = m->p.mu > 0.0 ? (float)m->p.mu : 0.0f;
  A.yield32 = (float)yield;
  for (int k = 0; k < HG_MAX_PLANES; ++k)
    for (int c = 0; c < 2; ++c) A.px[k][c] = (float)m->p.planes[k].x[c];
  auto kernel = m->p.basis == HG_BASIS_UGIMP ? k64_g2p<HG_BASIS_UGIMP> : k64_g2p<HG_BASIS_LINEAR>;
  const int t = point_threads(m);
  HG_LAUNCH_PDL(kernel, g2p_blocks(m, A.nn, t), t, 0, m->ctx->stream, m->p, A);
  HG_CHECK_LAUNCH();
  m->next_clear = true;
  return HG_OK;
}

} // namespace

// The accumulators of P2G (mass, momentum, force) are a pair: the last G2P
// cleared the other set, which becomes this step's.
hg_status mpm64_to_grid(hg_mpm *m) {
  cudaStream_t s = m->ctx->stream;
  const int64_t nn = (int64_t)(m->p.nx + 1) * (m->p.ny + 1);
  if (m->next_clear) {
    std::swap(m->g_mass.p, m->g_mass_next.p);
    std::swap(m->g_mom.p, m->g_mom_next.p);
    std::swap(m->g_force.p, m->g_force_next.p);
    m->next_clear = false;
  } else {
    HG_CUDA_TRY(cudaMemsetAsync(m->g_mass.p, 0, sizeof(double) * nn, s));
    HG_CUDA_TRY(cudaMemsetAsync(m->g_mom.p, 0, sizeof(double) * 2 * nn, s));
    HG_CUDA_TRY(cudaMemsetAsync(m->g_force.p, 0, sizeof(double) * 2 * nn, s));
  }
  if (m->n <= 0) return HG_OK;
  P2gArgs A;
  A.n = m->n;
  A.q = m->q.p;
  A.v = m->v.p;
  A.m = m->m.p;
  A.vol = m->vol.p;
  A.hl = m->hl.p;
  A.be = m->be.p;
  A.J = m->J.p;
  A.jh = m->jh.p;
  A.g_mass = m->g_mass.p;
  A.g_mom = m->g_mom.p;
  A.g_force = m->g_force.p;
  A.status = m->status.p;
  A.half_kappa = m->p.kappa * 0.5;
  auto kernel = m->p.basis == HG_BASIS_UGIMP ? k64_p2g<HG_BASIS_UGIMP> : k64_p2g<HG_BASIS_LINEAR>;
  const int t = point_threads(m);
  HG_LAUNCH_PDL(kernel, blocks_for(m->n, t), t, 0, s, m->p, A);
  HG_CHECK_LAUNCH();
  return HG_OK;
}

hg_status mpm64_step(hg_mpm *m, double dt) {
  hg_status st;
  if ((st = mpm64_to_grid(m)) || (st = grid_pass<true, true>(m, dt))) return st;
  return to_points(m, dt);
}

hg_status mpm64_phase0(hg_mpm *m) {
  cudaStream_t s = m->ctx->stream;
  const int64_t nn = (int64_t)(m->p.nx + 1) * (m->p.ny + 1);
  // clearRasterizedData (PhysicsGrid.cpp:107-114)
  HG_CUDA_TRY(cudaMemsetAsync(m->g_mom_new.p, 0, sizeof(double) * 2 * nn, s));
  HG_CUDA_TRY(cudaMemsetAsync(m->g_vel.p, 0, sizeof(double) * 2 * nn, s));
  HG_CUDA_TRY(cudaMemsetAsync(m->g_acc.p, 0, sizeof(double) * 2 * nn, s));
  return mpm64_to_grid(m);
}

hg_status mpm64_phase1(hg_mpm *m, double dt) { return grid_pass<true, false>(m, dt); }

hg_status mpm64_phase2(hg_mpm *m, double dt) {
  const hg_status st = grid_pass<false, true>(m, dt);
  return st != HG_OK ? st : to_points(m, dt);
}

} // namespace hg
