"""The bounding box's reduction: the first body holding an extreme value wins
(src/bounding_box.cpp:33-41), which shows in the sign of a zero, at the edges
of warps, blocks and the grid."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1000, 155648, 155649])
def test_first_extreme_wins(bh, n):
    rng = np.random.default_rng(n)
    pos = rng.choice([-0.0, 0.0, 1e-300, -1e-300, 3.0, -3.0], size=(n, 3), p=[0.2, 0.2, 0.15, 0.15, 0.15, 0.15])
    pos[:, 1] = rng.choice([0.0, -0.0], n)          # both extremes are zeros
    pos[:, 2] = np.where(rng.random(n) < 0.5, -0.0, -rng.random(n))  # the maximum is a zero, mostly
    with bh.Context(n) as c:
        c.set_bodies(pos, np.zeros((n, 3)), np.ones(n), np.arange(n, dtype=np.uint64))
        got = np.asarray(c.compute_bbox()).reshape(6)
    ax = np.arange(3)
    want = np.concatenate([pos[pos.argmin(axis=0), ax], pos[pos.argmax(axis=0), ax]])
    assert_bits_equal(got, want, f"bbox n={n}")
