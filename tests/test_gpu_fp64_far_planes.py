"""FP64 MPM with a tilted sliding plane given by a point far from the grid: the
nodes and points behind it are the reference's (PhysicsGrid.cpp:611-673,
MaterialPoints.cpp:371-423, both in FP64 from that point), whatever FP32 makes
of the distance. Against the CPU oracle over one step: 1e-12 relative on grid
fields and velocities, positions within 1e-15 m and four roundings at the
point's distance (the projection's difference of coordinates)."""
import numpy as np
import pytest

import oracle
import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("cells", [0.0, 1e4, 1e5, 1e6, 1e9])
@pytest.mark.parametrize("basis", [0, 1])
@pytest.mark.parametrize("bound", [-np.inf, -1e7 * H, 0.05])
def test_far_anchor_matches_oracle(ctx, cells, basis, bound):
    a = np.radians(37.3)  # no two of the grid's nodes lie alike to the plane
    n, along = np.array([np.sin(a), np.cos(a)]), np.array([-np.cos(a), np.sin(a)])
    x = np.array([0.1, 0.05]) + cells * H * along
    mat = scenes.mpm_material()
    args = (mat["shear_modulus"], mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"],
            scenes.GRAVITY)
    lo, hi = (0.0, 0.0), (0.25, 0.15)
    rng = np.random.default_rng(9)
    k = 4001
    vol = np.full(k, 0.25 * H * H)
    p = (rng.uniform([0.01, 0.01], [0.2, 0.12], (k, 2)), rng.normal(0.0, 0.3, (k, 2)),
         1550.0 * vol, vol, np.full(k, 0.25 * H))
    g = hg.MPM(ctx, lo, hi, H, *args, [(x, n, False, bound)], basis=basis, precision=hg.FP64,
               capacity=k)
    c = oracle.MPM(lo, hi, H, basis, *args)
    c.add_plane(x, n, False, bound)
    g.upload(*p)
    c.set_particles(*p)
    g.flow(1.0e-5, 1)
    c.step(1.0e-5, 1)
    G, C = g.grid(), c.grid()
    for f in ("mass", "mom", "mom_new", "force", "vel", "acc"):
        assert rel(G[f], C[f]) <= 1e-12, f
    P, Q = g.download(), c.particles()
    assert np.abs(P["q"] - Q["q"]).max() <= 1e-15 + 4.0 * 2.0 ** -53 * cells * H
    assert rel(P["v"], Q["v"]) <= 1e-12
    assert g.status() == 0
