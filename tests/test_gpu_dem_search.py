"""The DEM step's search, offsets and list order against the CPU oracle where
they can go wrong: bodies on either side of zero and far from it, lists longer
than the search keeps, a body that is the second of many contacts, sizes at
the edges of the emission pass's blocks and tiles, the one-thread-per-body
search of many bodies, and steps resumed after the bodies changed. FP64 steps
reproduce the reference's operations, so every comparison is for equality."""
import math

import numpy as np
import pytest

import oracle
import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu


def pair(ctx, q, v, r, fixed, planes=()):
    m = 2600.0 * math.pi * r * r
    p = scenes.dem_params()
    g = hg.DEM(ctx, scenes.GRAVITY, p["kn"], p["kt"], p["gamman"], p["gammat"], p["mu"], planes,
               capacity=len(r), contact_capacity=8 * len(r) + 64)
    g.upload(q, v, r, m, 0.5 * m * r * r, fixed)
    c = oracle.DEM(q, v, r, m, 0.5 * m * r * r, fixed, scenes.GRAVITY, p["kn"], p["kt"],
                   p["gamman"], p["gammat"], p["mu"], 1.0)
    for x, n in planes:
        c.add_plane(x, n)
    return g, c


def assert_same(g, c):
    (qg, vg), (qc, vc) = g.download(), c.state()
    assert np.array_equal(qg, qc)
    assert np.array_equal(vg, vc)
    rg, rc = g.contacts(), c.contacts()
    assert rg.shape == rc.shape and np.array_equal(rg, rc)
    assert g.status() == 0


def lattice(n, per_row, pitch=1.9e-3, x0=0.0, y0=0.0, seed=5):
    rng = np.random.default_rng(seed)
    k = np.arange(n)
    row, col = k // per_row, k % per_row
    q = np.zeros((n, 3))
    q[:, 0] = x0 + pitch * (col + 0.5 * (row % 2)) + rng.uniform(-5e-5, 5e-5, n)
    q[:, 1] = y0 + pitch * row * math.sqrt(0.75) + rng.uniform(-5e-5, 5e-5, n)
    v = rng.normal(0.0, 0.05, (n, 3))
    return q, v, rng.uniform(0.9e-3, 1.1e-3, n)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1025, 4097])
@pytest.mark.parametrize("x0,y0", [(-0.011, -0.007), (731.25, -1904.5)])
def test_lattice_around_and_far_from_zero(ctx, n, x0, y0):
    q, v, r = lattice(n, 31, x0=x0, y0=y0)
    fixed = np.zeros(n, dtype=np.uint8)
    fixed[::17] = 1
    v[::17] = 0.0
    g, c = pair(ctx, q, v, r, fixed, [((x0 - 2e-4, 0.0), (1.0, 0.0)), ((0.0, y0), (0.6, 0.8))])
    g.flow(1e-6, 3)
    c.step(1e-6, 3)
    assert_same(g, c)
    g.flow(1e-6, 20)  # replayed pairs of steps
    c.step(1e-6, 20)
    assert_same(g, c)


@pytest.mark.parametrize("big", [0, 13, 28])
@pytest.mark.parametrize("fixed_ring", [False, True])
def test_one_body_with_many_contacts(ctx, big, fixed_ring):
    """28 disks around one: as the first of its contacts more than the search
    keeps per body, as the second a long incoming list."""
    n, R, r1 = 29, 9.0e-3, 1.0e-3
    ring = np.delete(np.arange(n), big)
    a = 2.0 * math.pi * np.arange(28) / 28.0
    q, v = np.zeros((n, 3)), np.zeros((n, 3))
    q[ring, 0], q[ring, 1] = (R + r1 - 2e-5) * np.cos(a), (R + r1 - 2e-5) * np.sin(a)
    v[ring, 2] = np.linspace(-40.0, 40.0, 28)
    r = np.full(n, r1)
    r[big] = R
    fixed = np.zeros(n, dtype=np.uint8)
    if fixed_ring:
        fixed[ring[::2]] = 1
    g, c = pair(ctx, q, v, r, fixed)
    for k in (1, 6):
        g.flow(1e-6, k)
        c.step(1e-6, k)
        assert_same(g, c)
    assert len(g.contacts()) >= 28


def test_search_of_many_bodies(ctx):
    """Above 1,024 bodies per SM one thread searches all of a body's cells,
    and the tile sums take a pass of their own."""
    n = 180001
    q, v, r = lattice(n, 400)
    g, c = pair(ctx, q, v, r, np.zeros(n, dtype=np.uint8), [((0.0, 0.0), (0.0, 1.0))])
    g.flow(1e-6, 2)
    c.step(1e-6, 2)
    assert_same(g, c)


def test_steps_after_the_bodies_changed(ctx):
    n = 700
    q, v, r = lattice(n, 27)
    g, c = pair(ctx, q, v, r, np.zeros(n, dtype=np.uint8), [((0.0, 0.0), (0.0, 1.0))])
    for k in (5, 4, 1):
        g.flow(1e-6, k)
        c.step(1e-6, k)
        q2, v2 = c.state()
        q2[:, 0] += 2.5e-3  # a shift by more than a cell
        g.set_state(q2, v2)
        c.set_state(q2, v2)
    g.flow(1e-6, 1)
    c.step(1e-6, 1)
    assert_same(g, c)
    g.set_state(v=0.5 * v2)  # the positions, and their bins, stay
    c.set_state(v=0.5 * v2)
    g.flow(1e-6, 7)
    c.step(1e-6, 7)
    assert_same(g, c)
    # a checkpoint carries no list offsets: the history is searched by key
    h, _ = pair(ctx, q, v, r, np.zeros(n, dtype=np.uint8), [((0.0, 0.0), (0.0, 1.0))])
    h.load_state(g.state())
    h.flow(1e-6, 6)
    c.step(1e-6, 6)
    assert_same(h, c)
