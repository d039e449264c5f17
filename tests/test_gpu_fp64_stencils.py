"""The FP64 MPM and coupling kernels where their short forms hand over to the
general ones: half-widths at and beyond h / 2 and wider than the kernels'
stencils, points near the grid's edges, be_bar that is not symmetric, points
with J above 1, just homogenised or scripted, a sliding tilted plane; against
the CPU oracle at the FP64 path's tolerances (1e-12 relative on grid fields and
velocities, 1e-13 on J and be_bar, 1e-15 m on positions; the coupling's sums
1e-10)."""
import numpy as np
import pytest

import oracle
import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3
PLANES = [((0.0, 0.0), (0.0, 1.0), True, -np.inf), ((0.1, 0.02), (0.6, 0.8), False, 0.01)]


def rel(a, b):
    den = np.abs(b).max()
    return np.abs(a - b).max() / (den if den > 0 else 1.0)


def points(n, seed, hl, symmetric):
    rng = np.random.default_rng(seed)
    q = rng.uniform([-0.9 * H, -0.9 * H], [0.2, 0.1], (n, 2))
    q[:40, 0] = H * rng.integers(0, 30, 40)  # on node lines
    e, s = rng.uniform(-0.02, 0.02, n), rng.uniform(-0.02, 0.02, n)
    skew = 0.0 if symmetric else np.where(rng.random(n) < 0.3, 1e-3, 0.0)
    be = np.stack([1.0 + e, s + skew, s, (1.0 + s * s) / (1.0 + e)], axis=1)
    half = 0.25 * H
    vol = np.full(n, 4.0 * half * half)
    return dict(q=q, v=rng.normal(0.0, 0.3, (n, 2)), m=1550.0 * vol, vol=vol,
                hl=np.full(n, hl * H), be=be, J=rng.uniform(0.97, 1.02, n),
                jh=(rng.random(n) < 0.1).astype(np.int32),
                kin=(rng.random(n) < 0.05).astype(np.uint8))


def both(ctx, p, basis):
    # a grid that the widest stencils leave at none of the points
    lo, hi, mat = (-4 * H, -4 * H), (0.25, 0.15), scenes.mpm_material()
    args = (mat["shear_modulus"], mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"],
            scenes.GRAVITY)
    g = hg.MPM(ctx, lo, hi, H, *args, PLANES, basis=basis, precision=hg.FP64,
               capacity=len(p["m"]))
    c = oracle.MPM(lo, hi, H, basis, *args)
    for x, n, st, lb in PLANES:
        c.add_plane(x, n, st, lb)
    for o in (g.upload, c.set_particles):
        o(p["q"], p["v"], p["m"], p["vol"], p["hl"], p["be"], p["J"], p["jh"], p["kin"])
    return g, c


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("basis,hl", [(0, 0.25), (1, 0.15), (1, 0.25), (1, 0.5), (1, 0.7),
                                      (1, 1.0), (1, 1.6)])
def test_step_matches_oracle(ctx, basis, hl, symmetric):
    p = points(3001, 7, hl, symmetric)
    g, c = both(ctx, p, basis)
    for nsteps in (1, 2):
        g.flow(1.0e-5, nsteps)
        c.step(1.0e-5, nsteps)
        G, C = g.grid(), c.grid()
        for k in ("mass", "mom", "mom_new", "force", "vel", "acc"):
            assert rel(G[k], C[k]) <= 1e-12, k
        P, Q = g.download(), c.particles()
        assert np.abs(P["q"] - Q["q"]).max() <= 1e-15
        assert rel(P["v"], Q["v"]) <= 1e-12
        assert np.abs(P["J"] - Q["J"]).max() <= 1e-13
        assert np.abs(P["be"] - Q["be"]).max() <= 1e-13
        assert np.array_equal(P["jh"], Q["jh"])
    assert g.status() == 0


@pytest.mark.parametrize("basis,hl", [(0, 0.25), (1, 0.25), (1, 0.7), (1, 1.6)])
def test_coupling_matches_oracle(ctx, basis, hl):
    p = points(9001, 3, hl, True)
    p["jh"][:], p["kin"][:] = 0, 0
    g, c = both(ctx, p, basis)
    sc = scenes.dem_column(n=900, per_row=45, pitch=3.9e-3, rmin=1.8e-3, rmax=2.2e-3,
                           jitter=0.1e-3, x0=0.01, y0=0.02, rho=1550.0)
    sc["v"][:, 1] = -0.4
    sc["fixed"][:9] = 1
    dp, dem_planes = scenes.dem_params(kn=1e4), [((0.0, 0.0), (0.0, 1.0))]
    w = np.where(np.arange(900) % 4 == 0, 0.5, 1.0)
    args = (scenes.GRAVITY, dp["kn"], dp["kt"], dp["gamman"], dp["gammat"], dp["mu"])
    gd = hg.DEM(ctx, *args, dem_planes, capacity=900)
    gd.upload(sc["q"], sc["v"], sc["r"], sc["m"], sc["I"], sc["fixed"])
    cd = oracle.DEM(sc["q"], sc["v"], sc["r"], sc["m"], sc["I"], sc["fixed"], *args, 1.0)
    for x, n in dem_planes:
        cd.add_plane(x, n)
    gd.set_weights(w)
    cd.set_weights(w)
    gh, ch = hg.Hybrid(ctx, g, gd), oracle.Hybrid(c, cd)
    for _ in range(3):  # the exchange's grids alternate
        gh.step(1.0e-5, 1, True, True)
        ch.step(1.0e-5, 1, True, True)
        A, B = gh.coupling(), ch.coupling()
        assert len(B["packed_dem"]) > 100
        for k in ("packed_dem", "packed_mpm", "homog_factor"):
            assert np.array_equal(A[k], B[k]), k
        for k in ("dem_mass_grid", "dem_mom_grid", "v_after", "at_after", "homog_stress",
                  "homog_velocity"):
            assert rel(A[k], B[k]) <= 1e-10, k
        (qg, vg), (qc, vc) = gd.download(), cd.state()
        assert np.abs(qg - qc).max() <= 1e-15 and rel(vg, vc) <= 1e-10
        assert rel(g.download()["v"], c.particles()["v"]) <= 1e-10
