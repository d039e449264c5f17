"""Batches over the forms that their work queue and their kernel take (1,216 CTAs
on 152 SMs): fewer tiles than half of the CTAs, more tiles than CTAs, so many
that several are claimed at a time; as many members as the long passes have room
for and one more; a tile with one point more than a pass. Each member ends where it ends stepped alone, at the bounds of
test_gpu_batch."""
import numpy as np
import pytest

import libhybridgrains_gb300 as hg
from libhybridgrains_gb300 import scenes

pytestmark = pytest.mark.gpu

H, DT, STEPS = 5.0e-3, 1.0e-5, 20


def make(ctx, tiles, crowd, seed):
    """tiles x tiles tiles of six points each, crowd in one of them."""
    rng = np.random.default_rng(seed)
    t = np.stack(np.meshgrid(np.arange(tiles), np.arange(tiles)), axis=-1).reshape(-1, 1, 2)
    u = (16.0 * t + rng.uniform(0.5, 15.5, (tiles * tiles, 6, 2))).reshape(-1, 2)
    u = np.concatenate([u, 16.0 * (seed % tiles) + rng.uniform(0.5, 15.5, (crowd - 6, 2))])
    n = len(u)
    mat = scenes.mpm_material()
    m = hg.MPM(ctx, (0.0, 0.0), (16 * tiles * H,) * 2, H, mat["shear_modulus"],
               mat["bulk_modulus"], mat["dp_alpha"], mat["flip_alpha"], scenes.GRAVITY, [],
               capacity=n)
    vol = np.full(n, 0.02 * H * H)
    m.upload(u * H, rng.normal(0.0, 0.02, (n, 2)), 1550.0 * vol, vol, np.full(n, 0.05 * H))
    return m


@pytest.mark.parametrize("members,tiles,crowd", [
    (20, 4, 1025), (20, 8, 1025), (20, 16, 1025), (128, 2, 1153), (129, 2, 1025), (1, 2, 2305)])
def test_members_step_as_alone(ctx, members, tiles, crowd):
    alone = [make(ctx, tiles, crowd, k) for k in range(members)]
    together = [make(ctx, tiles, crowd, k) for k in range(members)]
    b = hg.Batch(ctx, max_members=members)
    for m in together:
        b.add(m, DT)
    for steps in (1, STEPS - 1):
        b.step(steps)
        for m in alone:
            m.flow(DT, steps)
    for t, a in zip(together, alone):
        T, A = t.download(), a.download()
        assert np.abs(T["q"] - A["q"]).max() <= 1e-9
        assert np.linalg.norm(T["v"] - A["v"]) <= 1e-5 * np.linalg.norm(A["v"])
        assert np.abs(T["J"] - A["J"]).max() <= 1e-6
        assert t.status() == 0
    b.close()
    for m in alone + together:
        m.close()
