"""The DEM step's bins and FP32 distance bounds against the FP64 tests.

A centre's cell and offset come from one fixed-point split (24 fraction bits
of x / H); radii are truncated to FP32. The search takes no pair whose FP32
distance exceeds ra + rb + tol, every pair below ra + rb - tol, and decides the
rest in FP64 (SpatialGrid.cpp:14-19, CircleGeometry.cpp:22-30,
ballBallCCDCollisionHappens with q0 == q1), with tol = 4e-6 of the cell width.
The arithmetic is restated with every operation rounded on its own, on pairs
placed within a few tol of contact, near and far from the origin."""
import numpy as np
import pytest

R0, R1 = 0.9e-3, 1.1e-3
H = 2.0 * R1 * (1.0 + 1.0e-6)
BIAS = 1.5 * 2.0 ** 28


def split(x):
    u = x * (1.0 / H) + BIAS
    k = u.view(np.int64) - np.float64(BIAS).view(np.int64)
    frac = (k & 0xFFFFFF).astype(np.float32) * np.float32(2.0 ** -24) * np.float32(H)
    return k >> 24, frac


def truncated(r):
    return (r.view(np.int64) & ~np.int64((1 << 29) - 1)).view(np.float64).astype(np.float32)


@pytest.mark.parametrize("reach", [0.05, 100.0, 4000.0])
def test_bounds_never_contradict_fp64(reach):
    rng = np.random.default_rng(7)
    n = 500_000
    tol = 4.0e-6 * H
    ra, rb = rng.uniform(R0, R1, n), rng.uniform(R0, R1, n)
    xa, ya = rng.uniform(-reach, reach, n), rng.uniform(-reach, reach, n)
    u = rng.uniform(-3.0, 3.0, n)
    u[: n // 10] = rng.choice([-1.0, 1.0], n // 10)
    d = ra + rb + u * tol
    phi = rng.uniform(0.0, 2.0 * np.pi, n)
    xb, yb = xa + d * np.cos(phi), ya + d * np.sin(phi)
    (cxa, oxa), (cya, oya), (cxb, oxb), (cyb, oyb) = map(split, (xa, ya, xb, yb))
    assert (np.abs(cxb - cxa) <= 1).all() and (np.abs(cyb - cya) <= 1).all()
    Hf, tolf = np.float32(H), np.float32(tol)
    ex = (cxb - cxa).astype(np.float32) * Hf + (oxb - oxa)
    ey = (cyb - cya).astype(np.float32) * Hf + (oyb - oya)
    d2 = ex * ex + ey * ey
    s = truncated(ra) + truncated(rb)
    reject, accept = d2 > (s + tolf) ** 2, d2 < (s - tolf) ** 2
    aabb = (xa + ra >= xb - rb) & (ya + ra >= yb - rb) & (xb + rb >= xa - ra) & (yb + rb >= ya - ra)
    ddx, ddy = xa - xb, ya - yb
    truth = aabb & ((ddx * ddx + ddy * ddy) - (ra + rb) * (ra + rb) <= 0.0)
    assert not (reject & truth).any() and not (accept & ~truth).any()
    assert 0.2 < (~reject & ~accept).mean() < 0.6  # what the FP64 tests decide
