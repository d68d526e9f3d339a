"""After replayed steps of a far-field form, what reads the tree's FP64 records
gets the current tree's, as it does after steps launched one kernel at a time."""
from __future__ import annotations

import pytest

from conftest import G, assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["MODE_FP32_FAR", "MODE_FP32_GROUP", "MODE_PLAIN_FP64"])
def test_invariants_between_replayed_steps(bh, mode):
    pos, vel, mass, ids = bh.generate_system(11, 3000, 0.1, 0.05)
    out = []
    for graphs in (True, False):
        with bh.Context(len(mass)) as c:
            c.set_step_graphs(graphs)
            c.set_bodies(pos, vel, mass, ids)
            t, got = 0.0, []
            for _ in range(3):
                t = c.step(86400.0 * 20, 1.05, G, 4, getattr(bh, mode), t)
                got.append(c.invariants(G, 0.5)["U"])
            got.append(c.export_tree()[3])
            out.append(got)
    for a, b in zip(*out):
        assert_bits_equal(a, b, mode)
