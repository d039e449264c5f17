"""A disk that touches more disks than a partner list holds: the step keeps 32
contacts of it and reports HG_STATUS_CELL_OVERFLOW, and what it keeps acts on
both bodies of each contact, also where the contacts found are more than the
contact buffers hold (those kept are not)."""
import numpy as np
import pytest

import libhybridgrains_gb300 as hg

pytestmark = pytest.mark.gpu


def crowded(ctx, precision, capacity, small):
    """A disk of radius 1 with `small` disks on its rim and, apart from it, a row
    of disks in a chain, numbered after them."""
    chain = 20
    n = 1 + small + chain
    q, r = np.zeros((n, 3)), np.full(n, 0.01)
    r[0] = 1.0
    a = 2.0 * np.pi * (np.arange(small) + 0.25) / small
    q[1:1 + small, 0], q[1:1 + small, 1] = 1.009 * np.cos(a), 1.009 * np.sin(a)
    q[1 + small:, 0], q[1 + small:, 1] = 3.0 + 0.019 * np.arange(chain), 0.5
    m = 1e3 * np.pi * r * r
    d = hg.DEM(ctx, (0.0, 0.0), 1e4, 2e3, 1.0, 1.0, 0.5, [], capacity=n,
               contact_capacity=capacity, precision=precision)
    d.upload(q, np.zeros((n, 3)), r, m, 0.5 * m * r * r, np.zeros(n, dtype=np.uint8))
    return d, m


@pytest.mark.parametrize("precision", [hg.FP64, hg.MIXED])
@pytest.mark.parametrize("small,capacity", [(100, 60), (100, 51), (200, 60), (100, 400), (20, 60)])
def test_kept_contacts_act_on_both_bodies(ctx, precision, small, capacity):
    d, m = crowded(ctx, precision, capacity, small)
    d.flow(1e-6, 1)
    c = d.contacts()
    kept = min(small, 32)
    pairs = c[:, 1:3].astype(int)
    assert len(pairs) == kept + 19
    assert (pairs[:kept, 0] == 0).all()
    assert d.status() == (0 if small <= 32 else 8)  # HG_STATUS_CELL_OVERFLOW
    _, v = d.download()
    # every body's velocity is that of its contacts' forces: fn + ft
    f = np.zeros((len(m), 2))
    np.add.at(f, pairs[:, 0], c[:, 17:19] + c[:, 19:21])
    np.add.at(f, pairs[:, 1], -(c[:, 17:19] + c[:, 19:21]))
    want = 1e-6 * f / m[:, None]
    assert (np.abs(want[pairs[:, 1]]).max(axis=1) > 0.0)[:kept].all()
    # FP64: a sum of at most 32 terms; MIXED: the same in FP32
    tol = 32.0 * (2.0 ** -53 if precision == hg.FP64 else 2.0 ** -23)
    scale = np.zeros((len(m), 1))
    for k in (0, 1):
        np.add.at(scale[:, 0], pairs[:, k], np.abs(c[:, 17:21]).sum(axis=1))
    assert (np.abs(v[:, :2] - want) <= 2.0 * tol * 1e-6 * scale / m[:, None]).all()
