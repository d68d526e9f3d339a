"""The FP64 walks at the sizes where their splits change.

The bit-exact walk at the sizes where its split changes (lanes per body: 32
below 6,384 bodies, 8, and 4 from 14,592 on, with 152 SMs), at partly
filled warps, with softening, at theta 0 and for a planar system, against the
oracle bit for bit.  The masked walks with one warp per group and with teams
of 16 (up to 9,728 bodies), 8 (24,320, FP32) and 4 (48,640 list, 87,552 group,
204,288 FP32): the list form with the oracle's interaction counts and within
its 1e-13, the FP32 forms' counts against the list form's and their
accelerations within the far field's FP32 rounding of a direct sum."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import G, assert_bits_equal

pytestmark = pytest.mark.gpu


def compare(bh, port, pos, vel, mass, ids, theta, soft2=0.0):
    with bh.Context(len(mass)) as c:
        c.set_bodies(pos, vel, mass, ids)
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, soft2, bh.MODE_PLAIN_FP64)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
        total = c.interaction_count()
    keys = port.keys(p, bb)
    tree = port.tree(keys, p, m)
    want, cnt = port.accelerations(tree, keys, p, theta, G, soft2, bb, count=True)
    assert_bits_equal(acc, want, f"accelerations n={len(mass)} theta={theta} soft2={soft2}")
    assert int(counts.sum()) == total == int(np.sum(cnt))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1001, 3647, 3648, 7295, 7297, 14591, 14593])
def test_sizes(bh, port, n):
    pos, vel, mass, ids = bh.generate_system(n, max(n, 10), 0.1, 0.05)
    compare(bh, port, pos[:n], vel[:n], mass[:n], ids[:n], 1.05)


@pytest.mark.parametrize("n", [3, 127, 129, 6383, 6385, 24320, 24321])
def test_shared_sums_and_records_ahead(bh, port, n):
    """Up to 6,383 bodies a block's warps share the sums of their four bodies
    (partly filled blocks among them), and up to 24,320 with 4 lanes to a body
    the evaluation loads the next step's records ahead."""
    pos, vel, mass, ids = bh.generate_system(n, max(n, 10), 0.1, 0.05)
    compare(bh, port, pos[:n], vel[:n], mass[:n], ids[:n], 1.05)


@pytest.mark.parametrize("n", [700, 5000, 9000, 16000])
@pytest.mark.parametrize("theta,soft2", [(0.4, 0.0), (1.05, 1e-6), (0.8, 1e-2), (2.0, 0.0)])
def test_angles_and_softening(bh, port, n, theta, soft2):
    pos, vel, mass, ids = bh.generate_system(3, n, 0.1, 0.0)
    compare(bh, port, pos, vel, mass, ids, theta, soft2)


def test_theta_zero(bh, port):
    pos, vel, mass, ids = bh.generate_system(4, 600, 0.0, 0.0)
    compare(bh, port, pos, vel, mass, ids, 0.0)


@pytest.mark.parametrize("n", [900, 15000])
def test_planar_offset_and_float_valued(bh, port, n):
    """z = 0 for every body (zero components), coordinates and masses that
    are FP32 values (significands ending in zeros: the IEEE fall-back), and a
    system far from the origin."""
    pos, vel, mass, ids = bh.generate_system(5, n, 0.1, 0.0)
    flat = pos.copy(); flat[:, 2] = 0.0
    compare(bh, port, flat, vel, mass, ids, 1.05)
    compare(bh, port, pos.astype(np.float32).astype(np.float64), vel, mass.astype(np.float32).astype(np.float64), ids,
            1.05)
    compare(bh, port, pos + np.array([2.0e4, -1.0e4, 3.0e3]), vel, mass, ids, 1.05)


@pytest.mark.parametrize("n,theta,soft2", [(1, 1.05, 0.0), (31, 1.05, 0.0), (3647, 1.05, 0.0), (9728, 0.7, 0.0),
                                           (9729, 1.05, 0.0), (29191, 1.05, 1e-6), (48640, 0.8, 0.0),
                                           (48641, 1.3, 0.0)])
def test_list_form(bh, port, n, theta, soft2):
    pos, vel, mass, ids = bh.generate_system(n, max(n, 10), 0.1, 0.05)
    with bh.Context(n) as c:
        c.set_bodies(pos[:n], vel[:n], mass[:n], ids[:n])
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, soft2, bh.MODE_FP64_LIST)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
    keys = port.keys(p, bb)
    want, cnt = port.accelerations(port.tree(keys, p, m), keys, p, theta, G, soft2, bb, count=True)
    assert np.array_equal(counts, cnt)
    scale = np.linalg.norm(want, axis=1, keepdims=True)
    assert np.all(np.abs(acc - want) <= 1e-13 * np.maximum(scale, 1e-300))


@pytest.mark.parametrize("n", [10, 33, 1000, 9728, 9729, 24320, 24321, 87552, 87553, 204288, 204289])
def test_fp32_forms(bh, n):
    """Each split gives the accelerations of a direct sum to the opening test's
    error (median below 1e-6 at theta 0.5) and its own interaction set: at
    theta 0 every far-field body of another leaf and every direct body once;
    at 0.5 the group form's counts are never below the per-body form's."""
    theta = 0.5
    pos, vel, mass, ids = bh.generate_system(n, n, 0.1, 0.0)
    with bh.Context(n) as c:
        c.set_bodies(pos, vel, mass, ids)
        c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        far = c.compute_accelerations(theta, G, 0.0, bh.MODE_FP32_FAR)
        far_counts = c.interaction_counts()
        assert c.interaction_count() == int(far_counts.sum())
        again = c.compute_accelerations(theta, G, 0.0, bh.MODE_FP32_FAR)
        group = c.compute_accelerations(theta, G, 0.0, bh.MODE_FP32_GROUP)
        group_counts = c.interaction_counts()
        sample = np.unique(np.linspace(0, n - 1, min(n, 256)).astype(np.int64))
        want = c.direct_sum(sample, G)
        if n <= 1000:
            leaves = c.tree_info()["leaves"]
            for mode in (bh.MODE_FP32_FAR, bh.MODE_FP32_GROUP):
                c.compute_accelerations(0.0, G, 0.0, mode)
                assert leaves == n and np.all(c.interaction_counts() == n - 1)
    assert_bits_equal(far, again, "a repeated call")
    assert np.all(group_counts >= far_counts)
    for acc in (far, group):
        err = np.linalg.norm(acc[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert np.median(err) < 1e-6 and np.all(err < 1e-3)
