"""A step that fails half-way leaves nothing behind that a later one adds to:
in the bounds-checking build each launch check of a step in turn reports an
error (on the host; the launches themselves are sound), the caller uploads its
state anew, and the steps after that are those of objects that never failed."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_hybrid_steps_after_a_failed_one():
    run("hybrid")


def test_small_mixed_scenes_after_a_failed_step():
    run("small")


def run(case):
    from libhybridgrains_gb300 import build
    build.build(bounds_check=True)
    env = dict(os.environ, HG_GPU_VARIANT="bounds")
    subprocess.run([sys.executable, os.path.abspath(__file__), case], env=env, check=True,
                   timeout=600)


def hybrid(hg, fail):
    """Both precisions of the bulk; sums compared at 1e-10 (order of FP64
    atomics) and, over an FP32 bulk, 1e-5."""
    from libhybridgrains_gb300 import scenes
    sc = scenes.dem_column(n=400, per_row=40, pitch=3.9e-3, rmin=1.8e-3, rmax=2.2e-3,
                           jitter=0.1e-3, x0=0.01, y0=0.02, rho=1550.0)
    sc["v"][:, 1] = -0.4
    rng = np.random.default_rng(5)
    n, h, mat, dp = 6000, 5.0e-3, scenes.mpm_material(), scenes.dem_params(kn=1e4)
    vol = np.full(n, 0.25 * h * h)
    pts = (rng.uniform([0.005, 0.005], [0.2, 0.1], (n, 2)), rng.normal(0.0, 0.3, (n, 2)),
           1550.0 * vol, vol, np.full(n, 0.25 * h))
    ctx = hg.Context(0)

    def objects(precision):
        m = hg.MPM(ctx, (-0.02, -0.02), (0.25, 0.15), h, mat["shear_modulus"], mat["bulk_modulus"],
                   mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY, [], basis=hg.UGIMP,
                   precision=precision, capacity=n)
        d = hg.DEM(ctx, scenes.GRAVITY, dp["kn"], dp["kt"], dp["gamman"], dp["gammat"], dp["mu"],
                   [((0.0, 0.0), (0.0, 1.0))], capacity=400)
        return m, d, hg.Hybrid(ctx, m, d)

    def upload(m, d, hy):
        m.upload(*pts)
        d.upload(sc["q"], sc["v"], sc["r"], sc["m"], sc["I"], sc["fixed"])
        hy.clear_homogenized()

    for precision, tol in ((hg.FP64, 1e-10), (hg.MIXED, 1e-5)):
        ref, got = objects(precision), objects(precision)
        upload(*ref)
        ref[2].step(1.0e-5, 2, True, True)
        want = ref[2].coupling()
        assert len(want["packed_dem"]) > 50
        upload(*got)
        got[2].step(1.0e-5, 3, True, True)
        failed = 0
        for k in range(1, 40):
            fail(k)
            try:
                got[2].step(1.0e-5, 1, True, True)
            except hg.HGError:
                failed += 1
            if fail(0) > 0:
                break  # the step has fewer checks
            upload(*got)
            got[2].step(1.0e-5, 2, True, True)
            have = got[2].coupling()
            for f in ("packed_dem", "packed_mpm", "homog_factor"):
                assert np.array_equal(have[f], want[f]), (k, f)
            for f in ("dem_mass_grid", "dem_mom_grid", "v_after", "at_after", "homog_stress",
                      "homog_velocity"):
                assert np.abs(have[f] - want[f]).max() <= tol * np.abs(want[f]).max(), (k, f)
        assert failed >= 8, failed


def small(hg, fail):
    """A MIXED scene stepped several steps in one launch each: the masses after
    a step are the points' to 1e-6 of the largest (FP32 sums)."""
    from libhybridgrains_gb300 import scenes
    rng = np.random.default_rng(6)
    n, h, mat = 3000, 5.0e-3, scenes.mpm_material()
    vol = np.full(n, 0.25 * h * h)
    pts = (rng.uniform([0.02, 0.02], [0.2, 0.1], (n, 2)), rng.normal(0.0, 0.3, (n, 2)),
           1550.0 * vol, vol, np.full(n, 0.25 * h))
    ctx = hg.Context(0)
    a, b = (hg.MPM(ctx, (0.0, 0.0), (0.25, 0.15), h, mat["shear_modulus"], mat["bulk_modulus"],
                   mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY, [], precision=hg.MIXED,
                   capacity=n) for _ in range(2))
    b.upload(*pts)
    b.flow(1.0e-5, 10)
    want = b.grid()["mass"]
    failed = 0
    for k in range(1, 40):
        a.upload(*pts)
        a.flow(1.0e-5, 1)
        fail(k)
        try:
            a.flow(1.0e-5, 10)
        except hg.HGError:
            failed += 1
        if fail(0) > 0:
            break
        a.upload(*pts)
        a.flow(1.0e-5, 10)
        assert np.abs(a.grid()["mass"] - want).max() <= 1e-6 * want.max(), k
    assert failed >= 10, failed


def main(case):
    sys.path.insert(0, ROOT)
    import libhybridgrains_gb300 as hg
    from libhybridgrains_gb300 import _capi
    fail = _capi.load().hg_check_fail_launch
    fail.argtypes, fail.restype = [ctypes.c_int64], ctypes.c_int64
    {"hybrid": hybrid, "small": small}[case](hg, fail)


if __name__ == "__main__":
    main(sys.argv[1])
