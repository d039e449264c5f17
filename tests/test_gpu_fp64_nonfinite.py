"""A point whose J is not a number (or infinite) in the FP64 MPM step: its nodes
get no finite force (no stress is 0 / J there, MaterialPoints.cpp:183-202), so
that the points around it follow, as on the CPU oracle; the status word says so.
What stays finite agrees at the FP64 path's 1e-12."""
import numpy as np
import pytest

import oracle
import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3


@pytest.mark.parametrize("basis", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("jh", [0, 1])
def test_reaches_the_nodes(ctx, basis, bad, jh):
    mat = scenes.mpm_material()
    args = (mat["shear_modulus"], mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"],
            scenes.GRAVITY)
    rng = np.random.default_rng(5)
    n = 800
    vol = np.full(n, 0.25 * H * H)
    J = rng.uniform(0.99, 1.0, n)
    J[17] = bad
    flag = np.zeros(n, dtype=np.int32)
    flag[17] = jh
    be = np.tile([1.0, 0.0, 0.0, 1.0], (n, 1))
    p = (rng.uniform([0.02, 0.02], [0.2, 0.1], (n, 2)), rng.normal(0.0, 0.1, (n, 2)),
         1550.0 * vol, vol, np.full(n, 0.25 * H), be, J, flag)
    lo, hi = (0.0, 0.0), (0.25, 0.15)
    g = hg.MPM(ctx, lo, hi, H, *args, [], basis=basis, precision=hg.FP64, capacity=n)
    c = oracle.MPM(lo, hi, H, basis, *args)
    g.upload(*p)
    c.set_particles(*p)
    g.flow(1.0e-5, 1)
    c.step(1.0e-5, 1)
    G, C = g.grid(), c.grid()
    P, Q = g.download(), c.particles()
    assert not np.isfinite(C["force"]).all()
    for a, b, keys in ((G, C, ("mass", "force", "vel", "acc")), (P, Q, ("q", "v"))):
        for k in keys:
            ok = np.isfinite(b[k])
            assert np.array_equal(np.isfinite(a[k]), ok), k
            assert np.abs(a[k][ok] - b[k][ok]).max() <= 1e-12 * np.abs(b[k][ok]).max(), k
    assert not np.isfinite(Q["q"]).all()
    assert g.status() != 0
    g.close()
