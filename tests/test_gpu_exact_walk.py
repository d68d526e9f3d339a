"""The FP64 walks at the sizes where their splits change.

The bit-exact walk at the sizes where its split changes (lanes per body:
32 below 3,648 bodies, 16, 8 and 4 from 14,592 on, with 152 SMs), at partly
filled warps, with softening, at theta 0 and for a planar system, against the
oracle bit for bit; the list form (the exact walk below 7,296 bodies, then 4,
8, 16 and 32 bodies per warp) with the oracle's interaction counts and within
its 1e-13."""
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


@pytest.mark.parametrize("n,theta,soft2", [(1, 1.05, 0.0), (3647, 1.05, 0.0), (7295, 0.7, 0.0), (7297, 1.05, 0.0),
                                           (14593, 1.05, 0.0), (29191, 1.05, 1e-6), (58367, 0.8, 0.0),
                                           (58369, 1.3, 0.0)])
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
