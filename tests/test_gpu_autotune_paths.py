"""The autotuner times the kernels that a launch shape is for: the two-kernel
steps, also on a scene small enough to step in one launch, which goes on doing
that; and what it chooses for a uGIMP scene, whose particle kernel takes no
shape, is no choice for a linear scene of that size."""
import numpy as np
import pytest

import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu


def column(ctx, npoints, basis=hg.LINEAR):
    cfg = scenes.serving_column(npoints, 1.5, 30.0)
    p = scenes.seed_column_points(cfg)
    pad = 0.02 if basis == hg.UGIMP else 0.0  # room for the points' extents
    m = hg.MPM(ctx, (-pad, -pad), cfg["grid_max"], cfg["h"], cfg["shear_modulus"],
               cfg["bulk_modulus"], cfg["dp_alpha"], cfg["flip_alpha"], scenes.GRAVITY,
               cfg["planes"], basis=basis, capacity=len(p["m"]))
    m.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"])
    return cfg, m


def launches(f):
    n = hg.kernel_launch_count()
    f()
    return hg.kernel_launch_count() - n


@pytest.mark.parametrize("npoints", [2000, 60000, 90000])
def test_the_two_kernels_are_timed(ctx, npoints):
    hg.tune_clear()
    cfg, m = column(ctx, npoints)
    m.flow(cfg["dt"], 1)
    steps = 16
    before = launches(lambda: m.flow(cfg["dt"], steps))
    n = launches(lambda: m.autotune(cfg["dt"], 5))
    # two launches a step, beside re-sorts
    assert n >= 2 * (4 * 6 + 16 * 48)
    assert before < 2 * steps if npoints < 75000 else before >= 2 * steps
    # afterwards as before (a re-sort may fall into either)
    after = min(launches(lambda: m.flow(cfg["dt"], steps)) for _ in range(3))
    assert after <= before
    assert m.status() == 0
    m.close()
    hg.tune_clear()


def test_ugimp_and_linear_classes_are_apart(ctx):
    hg.tune_clear()
    cfg, u = column(ctx, 60000, hg.UGIMP)
    r = u.autotune(cfg["dt"], 5)
    assert u.launch_shape() == r["chosen"]
    _, v = column(ctx, 60000, hg.UGIMP)
    v.flow(cfg["dt"], 1)
    assert v.launch_shape() == r["chosen"]
    _, m = column(ctx, 60000)
    m.flow(cfg["dt"], 1)
    assert m.launch_shape() == (0, 0)
    for x in (u, v, m):
        x.close()
    hg.tune_clear()
