"""The boundary pass and the child slots where their blocks change from
scanning the other blocks' sums themselves to a launch that does (128 blocks
of 1,024 boundaries for the summaries, 4,096 for the child counts): the tree
bit for bit against the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 131071, 131072, 4194304])
def test_tree_at_block_count_edges(bh, port, n):
    pos, vel, mass, ids = bh.generate_system(n, n, 0.1, 0.05)
    with bh.Context(n) as c:
        c.set_bodies(pos[:n], vel[:n], mass[:n], ids[:n])
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree(merge=False)
        got = c.export_tree()
        p, _, m, _, _ = c.get_bodies()
    tree = port.tree(port.keys(p, bb), p, m, merge=False)
    for a, b, name in zip(got, tree.records(), ("prefix", "depth", "mass", "com")):
        assert_bits_equal(a, b, f"n={n} {name}")
    tree.close()
