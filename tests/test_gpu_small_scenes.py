"""MIXED scenes stepped several steps per call, where one launch does a
whole step (small scenes) or tiles are cut into strips (a last round that leaves
CTAs idle): point counts on both sides of each choice, one to sixteen points per
cell, ragged columns, calls of one step to more than a chunk, re-sorts, points
that leave their tile's window. Against the FP64 path at the bounds that the
MIXED path has against the oracle over 20 steps (1e-9 m on positions, 1e-6 on J
and be_bar, 1e-4 relative on velocities; grid velocities 1e-5 and masses 1e-6
relative)."""
import numpy as np
import pytest

import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H = 5.0e-3


def column(wc, hc, ppc, x0, seed=2):
    """wc x hc cells from column x0, ppc = k^2 points per cell, in motion."""
    rng = np.random.default_rng(seed)
    k = int(round(np.sqrt(ppc)))
    off = (np.arange(k) + 0.5) / k
    gx, gy = np.meshgrid((np.arange(x0, x0 + wc)[:, None] + off).ravel(),
                         (np.arange(hc)[:, None] + off).ravel())
    q = np.stack([gx.ravel(), gy.ravel()], axis=1)
    n = len(q)
    q = (q + rng.uniform(-0.2, 0.2, (n, 2)) / k) * H
    vol = np.full(n, (H / k) ** 2)
    return dict(q=q, v=rng.normal(0.0, 0.02, (n, 2)), m=1550.0 * vol, vol=vol,
                hl=np.full(n, 0.5 * H / k))


def make(ctx, precision, nx, ny, n, planes=True, stiff=True):
    mat = scenes.mpm_material()
    k = 1.0 if stiff else 0.0
    pl = [((0.0, 0.0), (0.0, 1.0), True, -np.inf), ((nx * H, 0.0), (-1.0, 0.0), False, -np.inf)]
    return hg.MPM(ctx, (0.0, 0.0), (nx * H, ny * H), H, k * mat["shear_modulus"],
                  k * mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY,
                  pl if planes else [], precision=precision, capacity=n)


def same(a, b, steps_so_far, mass=1e-6):
    A, B = a.download(), b.download()
    assert np.abs(A["q"] - B["q"]).max() <= 1e-9
    assert np.abs(A["J"] - B["J"]).max() <= 1e-6
    assert np.abs(A["be"] - B["be"]).max() <= 1e-6
    assert np.linalg.norm(A["v"] - B["v"]) <= 1e-4 * np.linalg.norm(B["v"])
    G, F = a.grid(), b.grid()
    act = F["mass"] > 0
    assert np.abs(G["mass"] - F["mass"]).max() <= mass * F["mass"].max()
    if steps_so_far == 1:
        d = np.linalg.norm(G["vel"][act] - F["vel"][act])
        assert d <= 1e-5 * np.linalg.norm(F["vel"][act])
    assert a.status() == 0 and b.status() == 0


# strips of a quarter, of half a tile, whole tiles in a round; points at and
# above the limit; the two-launch path's quarters, halves, two rounds with a cut
# second one, and without
@pytest.mark.parametrize("wc,hc,ppc,x0", [
    (1, 1, 1, 15), (17, 9, 4, 7), (40, 80, 4, 20), (61, 67, 16, 3), (125, 150, 4, 0),
    (151, 125, 4, 5), (250, 300, 1, 9), (160, 200, 1, 2), (150, 200, 4, 0), (200, 260, 4, 1),
    (320, 420, 4, 6), (300, 340, 4, 0)])
def test_several_steps_per_call_match_fp64(ctx, wc, hc, ppc, x0):
    p = column(wc, hc, ppc, x0)
    n = len(p["m"])
    objs = [make(ctx, prec, x0 + wc + 13, hc + 11, n) for prec in (hg.MIXED, hg.FP64)]
    for o in objs:
        o.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"])
    done = 0
    for steps in (1, 4, 3, 12):
        for o in objs:
            o.flow(2.0e-5, steps)
        done += steps
        same(*objs, done)


def test_chunks_and_single_steps_mix(ctx):
    """Chunks, the steps after them, re-sorts in between and single steps, on one
    object; the same steps one call each on another."""
    p = column(45, 61, 4, 11)
    n = len(p["m"])
    a, b, f = (make(ctx, prec, 96, 80, n) for prec in (hg.MIXED, hg.MIXED, hg.FP64))
    for o in (a, b, f):
        o.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"])
    for steps in (16, 1, 21, 2, 7):
        a.flow(2.0e-5, steps)
        f.flow(2.0e-5, steps)
        for _ in range(steps):
            b.flow(2.0e-5, 1)
    A, B, F = (o.download() for o in (a, b, f))
    for X in (A, B):  # 47 steps: the 20-step bounds, by steps
        assert np.abs(X["q"] - F["q"]).max() <= 2.5e-9
        assert np.abs(X["J"] - F["J"]).max() <= 2.5e-6
        assert np.linalg.norm(X["v"] - F["v"]) <= 2.5e-4 * np.linalg.norm(F["v"])
    assert a.status() == 0 and b.status() == 0


def test_fast_points_leave_their_windows(ctx):
    """Points without stiffness at 0.2 cells per step, clusters one behind the
    other in two bands that pass each other: they cross tiles within a chunk, add
    to nodes outside the active tiles and enter tiles that others have left.
    Bound: FP32 velocities over 0.2 cells a step."""
    rng = np.random.default_rng(5)
    n = 400
    band = np.arange(n) % 2
    q = np.stack([0.1 + 0.1 * (np.arange(n) // 2 % 4) + rng.uniform(0.0, 0.02, n),
                  0.3 + 0.3 * band + rng.uniform(0.0, 0.02, n)], axis=1)
    q[band == 1, 0] += 0.4
    v = np.where(band == 0, 1.0, -1.0)[:, None] * np.array([[2.0, 0.0]])
    m, vol, hl = np.full(n, 1e-3), np.full(n, 1e-6), np.full(n, 1.25e-3)
    a, f = (make(ctx, prec, 200, 200, n, planes=False, stiff=False)
            for prec in (hg.MIXED, hg.FP64))
    for o in (a, f):
        o.upload(q, v, m, vol, hl)
        for steps in (40, 9, 32, 16):
            o.flow(5.0e-4, steps)
    assert np.abs(a.download()["q"] - f.download()["q"]).max() <= 97 / 40 * 2e-8
    assert a.status() == 0
    assert a.rebin_count() >= 2


@pytest.mark.parametrize("n", [1, 127, 129, 4001])
@pytest.mark.parametrize("hl", [0.03, 0.25, 0.4375, 0.5])
def test_ugimp_weights_at_their_joints_match_fp64(ctx, n, hl):
    """MIXED with the uGIMP basis on both sides of where a node's weight changes
    its form (points about +-hl and half-way around a node, on nodes) and at the
    first and last node that a point may touch, against the FP64 path: masses
    and momenta 1e-6 of the largest, positions 1e-12 m after one step and J 1e-6
    (the MIXED path's bounds for one step)."""
    rng = np.random.default_rng(8)
    # (not on +-hl: whether a node of weight 0 there is touched is rounding, and
    # what it adds to the gradient, force over mass, does not go to 0 with it)
    near = hl + np.array([-1e-2, 1e-2])
    joints = np.concatenate([[0.0, 0.5, -0.5, 0.5 * hl, 0.3], near, -near])
    lo, hi = 1, 39  # nodes whose neighbours are on the 40-cell grid
    u = rng.integers(lo, hi + 1, (n, 2)) + joints[rng.integers(0, len(joints), (n, 2))]
    u = np.clip(u, hl + 1e-3, 40.0 - hl - 1e-3)  # no point moves off the grid
    q = u * H
    vol = np.full(n, (2.0 * hl * H) ** 2)
    e = rng.uniform(-0.01, 0.0, n)
    be = np.stack([1.0 + e, np.zeros(n), np.zeros(n), 1.0 / (1.0 + e)], axis=1)
    p = dict(q=q, v=rng.normal(0.0, 0.1, (n, 2)), m=1550.0 * vol, vol=vol,
             hl=np.full(n, hl * H), be=be, J=1.0 + rng.uniform(-0.01, 0.0, n))
    mat = scenes.mpm_material()
    out = []
    for prec in (hg.MIXED, hg.FP64):
        o = hg.MPM(ctx, (0.0, 0.0), (40 * H, 40 * H), H, mat["shear_modulus"],
                   mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY, [],
                   basis=hg.UGIMP, precision=prec, capacity=n)
        o.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"], p["be"], p["J"])
        o.flow(1.0e-6, 1)
        assert o.status() == 0
        out.append((o.download(), o.grid()))
    (A, G), (B, F) = out
    assert np.abs(A["q"] - B["q"]).max() <= 1e-12
    assert np.abs(A["J"] - B["J"]).max() <= 1e-6
    assert np.abs(A["be"] - B["be"]).max() <= 1e-6
    assert np.abs(G["mass"] - F["mass"]).max() <= 1e-6 * F["mass"].max()
    for a, b in ((G["mass"][:, None] * G["vel"], F["mass"][:, None] * F["vel"]),):
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max() + 1e-6 * F["mass"].max() * 0.1


def plain(ctx, precision, n, nx=41, ny=37):
    return hg.MPM(ctx, (0.0, 0.0), (nx * H, ny * H), H, 1.0e3, 1.0e3, 0.0, 0.95, scenes.GRAVITY,
                  [], precision=precision, capacity=max(n, 1))


@pytest.mark.parametrize("n", [1, 5, 257, 5000])
def test_sort_keys_at_the_grid_edges(ctx, n):
    """Points on cell lines, on the grid's far edges (which belong to the last
    cell), in its first column and next to lines by one unit in the last place:
    the masses that the first step rasterises are those of the bilinear weights
    (1e-6 of the largest)."""
    rng = np.random.default_rng(3)
    x = np.concatenate([[0.0, 41.0, 1.0, 16.0, 40.0], 41.0 * rng.random(n)])[:n]
    y = np.concatenate([[37.0, 37.0, 0.0, 16.0, 32.0], 37.0 * rng.random(n)])[:n]
    k = rng.random((2, n)) < 0.3
    x, y = np.where(k[0], np.round(x), x), np.where(k[1], np.round(y), y)
    k = rng.random((2, n)) < 0.2
    x, y = np.where(k[0], np.nextafter(x, 0.0), x), np.where(k[1], np.nextafter(y, 0.0), y)
    q = np.minimum(np.stack([x, y], axis=1) * H, [41 * H, 37 * H])
    m = rng.uniform(1.0, 2.0, n)
    o = plain(ctx, hg.MIXED, n)
    o.upload(q, np.zeros((n, 2)), m, np.full(n, 1e-6), np.full(n, 0.25 * H))
    assert np.abs(o.download()["q"] - q).max() <= 1e-12  # the scatter keeps every point's place
    assert o.status() == 0  # (the step takes the points on the low edge off the grid)
    o.flow(1e-9, 1)
    u = q / H
    c = np.minimum(np.floor(u).astype(int), [40, 36])
    f = u - c
    mass = np.zeros((38, 42))
    for dx in (0, 1):
        for dy in (0, 1):
            w = (f[:, 0] if dx else 1.0 - f[:, 0]) * (f[:, 1] if dy else 1.0 - f[:, 1])
            np.add.at(mass, (c[:, 1] + dy, c[:, 0] + dx), w * m)
    got = np.asarray(o.grid()["mass"]).reshape(38, 42)
    assert np.abs(got - mass).max() <= 1e-6 * mass.max()


@pytest.mark.parametrize("bad", [-1e-3, 42.0, np.nan, np.inf, -np.inf, 1e300])
def test_points_off_the_grid_are_reported(ctx, bad):
    q = np.full((40, 2), 5.5 * H)
    q[17, 1] = bad * H
    o = plain(ctx, hg.MIXED, 40)
    o.upload(q, np.zeros((40, 2)), np.ones(40), np.full(40, 1e-6), np.full(40, 0.25 * H))
    assert o.status() & 2


def test_tiles_that_drop_out_are_cleared(ctx):
    n = 300
    rng = np.random.default_rng(4)
    o = plain(ctx, hg.MIXED, n, 200, 100)
    for x0 in (3.0, 150.0, 60.0):
        q = (rng.random((n, 2)) * 10.0 + [x0, 40.0]) * H
        o.upload(q, np.zeros((n, 2)), np.ones(n), np.full(n, 1e-6), np.full(n, 0.25 * H))
        o.flow(1e-9, 17)
        mass = np.asarray(o.grid()["mass"]).reshape(101, 201)
        assert abs(mass.sum() - n) <= 1e-5 * n
        assert np.all(mass[:, : int(x0)] == 0.0) and np.all(mass[:, int(x0) + 12:] == 0.0)


@pytest.mark.parametrize("per_tile", [1152, 1153, 2304, 5000])
@pytest.mark.parametrize("batched", [False, True])
def test_crowded_tiles_match_fp64(ctx, per_tile, batched):
    """Tiles with as many points as a pass takes, one more, two passes and more,
    one cell with more points than a pass, empty cells between: one step and
    five, against the FP64 path at the MIXED bounds, masses at 3e-6 (1,500 terms
    added up in FP32: sqrt(1500) 2^-24 = 2.3e-6)."""
    rng = np.random.default_rng(6)
    u = np.concatenate([rng.random((per_tile, 2)) * [15.9, 15.9] + [16.0, 16.0],
                        rng.random((1500, 2)) * 0.98 + [40.01, 20.01],
                        rng.random((700, 2)) * [30.0, 3.0] + [50.0, 20.0]])
    u[(np.floor(u[:, 0]) % 5 == 3) & (u[:, 0] < 32.0)] -= [1.0, 0.0]
    n = len(u)
    vol = np.full(n, 0.02 * H * H)
    args = (u * H, rng.normal(0.0, 0.02, (n, 2)), 1550.0 * vol, vol, np.full(n, 0.05 * H))
    a, f = (make(ctx, prec, 96, 64, n) for prec in (hg.MIXED, hg.FP64))
    a.upload(*args)
    f.upload(*args)
    done = 0
    b = hg.Batch(ctx, max_members=1) if batched else None
    if b:
        b.add(a, 1.0e-5)
    for steps in (1, 4):
        b.step(steps) if b else [a.flow(1.0e-5, 1) for _ in range(steps)]
        f.flow(1.0e-5, steps)
        done += steps
        same(a, f, done, 3e-6)
