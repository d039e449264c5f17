"""The FP64 MPM step at the ends of the material's range: no shear modulus, no
bulk modulus, no friction. Without a shear modulus mu |dev be| never exceeds
the yield stress (ConstitutiveModel.cpp:26-81), so be_bar keeps its deviator
whatever J is; without a yield stress every deviator is removed. Against the CPU
oracle at the FP64 path's tolerances (1e-12 relative on grid fields and
velocities, 1e-13 on J and be_bar, 1e-15 m on positions)."""
import numpy as np
import pytest

import oracle
import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3


def rel(a, b):
    den = np.abs(b).max()
    return np.abs(a - b).max() / (den if den > 0 else 1.0)


@pytest.mark.parametrize("basis", [0, 1])
@pytest.mark.parametrize("mu,kappa,alpha", [(0.0, 1.0, 1.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0),
                                            (0.0, 0.0, 0.0), (1.0, 0.0, 1.0), (1.0, 1.0, 0.0),
                                            (1e-12, 1.0, 1.0), (1.0, 1e-12, 1.0)])
def test_step_matches_oracle(ctx, mu, kappa, alpha, basis):
    """mu, kappa, alpha in units of the column's."""
    mat = scenes.mpm_material()
    args = (mu * mat["shear_modulus"], kappa * mat["bulk_modulus"], alpha * mat["dp_alpha"],
            mat["flip_alpha"], scenes.GRAVITY)
    rng = np.random.default_rng(21)
    n = 2001
    e, s = rng.uniform(-0.02, 0.02, n), rng.uniform(-0.02, 0.02, n)
    e[:50], s[:50] = 0.0, 0.0  # no deviator
    be = np.stack([1.0 + e, s, s, (1.0 + s * s) / (1.0 + e)], axis=1)
    vol = np.full(n, 0.25 * H * H)
    p = (rng.uniform([0.01, 0.01], [0.2, 0.1], (n, 2)), rng.normal(0.0, 0.3, (n, 2)), 1550.0 * vol,
         vol, np.full(n, 0.25 * H), be, rng.uniform(0.97, 1.03, n))
    lo, hi = (0.0, 0.0), (0.25, 0.15)
    g = hg.MPM(ctx, lo, hi, H, *args, [], basis=basis, precision=hg.FP64, capacity=n)
    c = oracle.MPM(lo, hi, H, basis, *args)
    g.upload(*p)
    c.set_particles(*p)
    for nsteps in (1, 3):
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
    assert g.status() == 0
