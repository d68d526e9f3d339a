"""The FP64 walks where FP32 squares of distances overflow (separations above
1.8e19, galactic distances in metres) or underflow: the opening tests the FP32
bounds cannot take are FP64's, so the accelerations are the oracle's bit for bit
in the plain form at each of its splits and in the LET forces, and the list
form has its interaction counts."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import G, assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 9000, 16000])
@pytest.mark.parametrize("span", [1e18, 1.2e19, 3e19, 5e20])
@pytest.mark.parametrize("theta", [0.3, 0.5, 1.05])
def test_plain_form(bh, port, n, span, theta):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, span, (n, 3))
    mass = 10.0 ** rng.uniform(25.0, 31.0, n)
    ids = np.arange(n, dtype=np.uint64)
    with bh.Context(n) as c:
        c.set_bodies(pos, np.zeros((n, 3)), mass, ids)
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, 0.0, bh.MODE_PLAIN_FP64)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
    keys = port.keys(p, bb)
    want, cnt = port.accelerations(port.tree(keys, p, m), keys, p, theta, G, 0.0, bb, count=True)
    assert np.array_equal(counts, cnt)
    assert_bits_equal(acc, want, f"accelerations n={n} span={span} theta={theta}")


# (a team of 16, of 4, and one warp to a group)
@pytest.mark.parametrize("n", [700, 9800, 49000])
@pytest.mark.parametrize("span", [1e-15, 1e-13, 1.2e19, 3e19, 5e20])
@pytest.mark.parametrize("theta", [0.4, 1.05])
def test_list_form(bh, port, n, span, theta):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, span, (n, 3))
    pos[: n // 4] = pos[0] + (pos[: n // 4] - pos[0]) * 1e-4  # close pairs
    mass = 10.0 ** rng.uniform(25.0, 31.0, n)
    with bh.Context(n) as c:
        c.set_bodies(pos, np.zeros((n, 3)), mass, np.arange(n, dtype=np.uint64))
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, 0.0, bh.MODE_FP64_LIST)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
    keys = port.keys(p, bb)
    want, cnt = port.accelerations(port.tree(keys, p, m), keys, p, theta, G, 0.0, bb, count=True)
    assert np.array_equal(counts, cnt)
    # some 1,000 terms and as many additions, to a few roundings each, against
    # the terms' magnitudes (taken from the direct sum)
    for i in range(0, n, n // 50):
        r = np.linalg.norm(p - p[i], axis=1)
        with np.errstate(divide="ignore"):
            terms = np.where(r > 0, G * m / (r * r), 0.0).sum()
        assert np.linalg.norm(acc[i] - want[i]) <= 5e-13 * terms


@pytest.mark.parametrize("span", [1.2e19, 5e20])
@pytest.mark.parametrize("direct", [False, True])
def test_let_forces(bh, port, span, direct):
    n, theta = 3000, 0.5
    rng = np.random.default_rng(7)
    pos = rng.uniform(0.0, span, (n, 3))
    mass = 10.0 ** rng.uniform(25.0, 31.0, n)
    bb = port.bbox(pos)
    keys = port.keys(pos, bb)
    near = keys < np.uint64(1 << 62)
    sk, sp, sm, _, _, _ = port.sort(keys[near], pos[near], mass[near], np.zeros((n, 3))[near],
                                    np.arange(n, dtype=np.uint64)[near])
    # the other bodies as records of depth-4 cells
    cell, inv = np.unique(keys[~near] >> np.uint64(63 - 12) << np.uint64(63 - 12), return_inverse=True)
    m = np.bincount(inv, mass[~near])
    com = np.stack([np.bincount(inv, mass[~near] * pos[~near][:, a]) for a in range(3)], 1) / m[:, None]
    rec = (cell.astype(np.uint64), np.full(len(cell), 4, np.uint8), m, np.ascontiguousarray(com))
    tree = port.tree(sk, sp, sm, merge=False)
    want = port.let_accelerations(tree, rec, sk, sp, theta, G, bb, direct=direct)
    tree.close()
    k = len(sm)
    with bh.Context(k) as c:
        c.set_bodies(pos[near], np.zeros((k, 3)), mass[near], np.arange(n, dtype=np.uint64)[near])
        c.set_bbox(bb); c.compute_keys(); c.sort_bodies(); c.build_tree(merge=False)
        got = c.let_accelerations(*rec, theta=theta, G=G, direct=direct)
    assert_bits_equal(got, want, f"LET forces span={span} direct={direct}")
