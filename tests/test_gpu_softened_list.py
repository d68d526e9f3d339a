"""The list form with softening: the reference's opening test includes it, so
the interaction counts are the oracle's, and the accelerations are within the
list form's accuracy, for softenings from far below the cells' sizes to far
above them, on both sides of each split into teams (16 warps to a group up to
4,864 bodies with softening, 8 up to 9,728, 4 up to 48,640, then one)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 700, 4864, 4865, 9728, 9729, 49000])
@pytest.mark.parametrize("theta,soft2", [(1.05, 0.0), (1.05, 1e-12), (0.8, 1e-4), (1.05, 1e-2), (0.8, 1.0), (1.05, 100.0)])
def test_counts_and_accelerations(bh, port, n, theta, soft2):
    pos, vel, mass, ids = bh.generate_system(n, max(n, 10), 0.1, 0.05)
    pos, vel, mass, ids = pos[:n], vel[:n], mass[:n], ids[:n]
    with bh.Context(n) as c:
        c.set_bodies(pos, vel, mass, ids)
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, soft2, bh.MODE_FP64_LIST)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
    keys = port.keys(p, bb)
    want, cnt = port.accelerations(port.tree(keys, p, m), keys, p, theta, G, soft2, bb, count=True)
    assert np.array_equal(counts, cnt)
    scale = np.linalg.norm(want, axis=1, keepdims=True)
    assert np.all(np.abs(acc - want) <= 1e-13 * np.maximum(scale, 1e-300))
