"""A point outside the grid is skipped and reported, and costs itself alone:
the other points of its tile and the nodes' masses and momenta are those of the
FP64 path, in every form of the MIXED kernels (a step in one launch on strips,
two launches over whole tiles, over strips, over tiles of several passes, a
batch). Bounds: the MIXED path's over 20 steps (1e-9 m on positions, 1e-6 on J
and be_bar, 1e-4 relative on velocities), masses 3e-6 of the largest (a node's
up to 4 x 16 terms in FP32 and the crowded case's 1,500: sqrt(1500) 2^-24)."""
import numpy as np
import pytest

import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3


def column(wc, hc, ppc, x0, seed=12):
    rng = np.random.default_rng(seed)
    k = int(round(np.sqrt(ppc)))
    off = (np.arange(k) + 0.5) / k
    gx, gy = np.meshgrid((np.arange(x0, x0 + wc)[:, None] + off).ravel(),
                         (np.arange(1, hc + 1)[:, None] + off).ravel())
    q = np.stack([gx.ravel(), gy.ravel()], axis=1)
    n = len(q)
    q = (q + rng.uniform(-0.2, 0.2, (n, 2)) / k) * H
    vol = np.full(n, (H / k) ** 2)
    return dict(q=q, v=rng.normal(0.0, 0.02, (n, 2)), m=1550.0 * vol, vol=vol,
                hl=np.full(n, 0.5 * H / k))


def make(ctx, precision, nx, ny, n):
    mat = scenes.mpm_material()
    return hg.MPM(ctx, (0.0, 0.0), (nx * H, ny * H), H, mat["shear_modulus"], mat["bulk_modulus"],
                  mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY,
                  [((0.0, 0.0), (0.0, 1.0), True, -np.inf)], precision=precision, capacity=n)


# one launch a step: quarter strips of one pass and of several; two launches:
# quarter strips of a turn per thread, whole tiles of 1,024 points and of 2,304
# (a batch takes each as whole tiles)
@pytest.mark.parametrize("wc,hc,ppc", [(61, 67, 16), (33, 40, 49), (150, 200, 4), (300, 340, 4),
                                       (256, 208, 9)])
@pytest.mark.parametrize("batched", [False, True])
def test_an_off_grid_point_costs_itself_alone(ctx, wc, hc, ppc, batched):
    x0 = 16
    p = column(wc, hc, ppc, x0)
    n, nx, ny = len(p["m"]), x0 + wc + 13, hc + 11
    # one below the grid at the left of a tile, one above it, one to the right,
    # one that is no number: each sorted into a cell of the grid's edge or its
    # corner, where tiles with points are; each first in its thread's turns
    bad = np.array([5, n // 3, n // 2, n - 7])
    p["q"][bad] = np.array([[16.2, -0.7], [17.3, -2.0], [x0 + wc / 2.0, -0.3], [33.1, -1e9]]) * H
    objs = [make(ctx, prec, nx, ny, n) for prec in (hg.MIXED, hg.FP64)]
    for o in objs:
        o.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"])
    a, f = objs
    b = hg.Batch(ctx, max_members=1) if batched else None
    if b:
        b.add(a, 1.0e-5)
    good = np.setdiff1d(np.arange(n), bad)
    for steps in (1, 8, 11):
        b.step(steps) if b else a.flow(1.0e-5, steps)
        f.flow(1.0e-5, steps)
        A, F = a.download(), f.download()
        assert np.array_equal(F["q"][bad], p["q"][bad]) and np.array_equal(A["v"][bad], F["v"][bad].astype(np.float32))
        assert np.abs(A["q"] - F["q"])[good].max() <= 1e-9
        assert np.abs(A["J"] - F["J"])[good].max() <= 1e-6
        assert np.abs(A["be"] - F["be"])[good].max() <= 1e-6
        assert np.linalg.norm((A["v"] - F["v"])[good]) <= 1e-4 * np.linalg.norm(F["v"][good])
        G, K = a.grid(), f.grid()
        assert np.abs(G["mass"] - K["mass"]).max() <= 3e-6 * K["mass"].max()
        assert abs(G["mass"].sum() - p["m"][good].sum()) <= 1e-6 * p["m"].sum()
        assert a.status() == 2 and f.status() == 2  # HG_STATUS_OUT_OF_GRID
    if b:
        b.close()
