"""The masked walks' teams where their shared stack would grow longest: systems
whose every popped range holds eight nodes that are opened in turn, round after
round, so that the ranges waiting pile up past the stack's 2,048."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import G

pytestmark = pytest.mark.gpu

POP = 4     # ranges a warp takes per round
STACK = 2048


def piled_up(team, rounds):
    """Leaf paths (octants from the root) of a system walked at theta 0 by a
    team: all ranges the next round takes from the stack's top are of eight
    nodes with eight children each, for `rounds` rounds after the third level;
    all others end in two leaves.  Also the most ranges the stack holds."""
    stack, leaves, r, most = [[()]], [], 0, 1
    while stack:
        taken = [stack.pop() for _ in range(min(len(stack), POP * team))]
        nodes = [nd for rng in taken for nd in rng]
        r += any(nd is not None and len(nd) >= 3 for nd in nodes)
        for k, nd in enumerate(nodes):
            if nd is None:
                continue
            if len(nd) < 3 or (r <= rounds and len(nodes) - k <= POP * team and len(nd) < 20):
                stack.append([nd + (o,) for o in range(8)])
            else:
                leaves += [nd + (0,), nd + (7,)]
                stack.append([None, None])
        most = max(most, len(stack))
    return leaves, most


def bodies(leaves, n):
    """n bodies: one at the centre of the first depth-21 cell of each leaf, two
    that span the box, and the rest on top of the first."""
    cells = np.zeros((len(leaves) + 1, 3), np.int64)
    for i, path in enumerate(leaves):
        for d, o in enumerate(path):
            for a in range(3):
                cells[i, a] |= ((o >> a) & 1) << (20 - d)
    cells[-1] = (1 << 21) - 1
    pos = (cells + 0.5) / 2.0 ** 21
    pos = np.concatenate([pos, [[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]])
    assert len(pos) <= n
    return np.concatenate([pos, np.repeat(pos[:1], n - len(pos), axis=0)])


# team, rounds of piling up, bodies, form
@pytest.mark.parametrize("team,rounds,n,mode", [(8, 8, 4612, "list"), (16, 5, 9728, "far"), (16, 4, 5000, "group"),
                                                (8, 8, 9729, "far"), (8, 9, 24320, "group")])
def test_full_stack(bh, team, rounds, n, mode):
    leaves, most = piled_up(team, rounds)
    assert most > STACK
    pos = bodies(leaves, n)
    rng = np.random.default_rng(n)
    mass = 10.0 ** rng.uniform(12.0, 20.0, n)
    mode = {"list": bh.MODE_FP64_LIST, "far": bh.MODE_FP32_FAR, "group": bh.MODE_FP32_GROUP}[mode]
    with bh.Context(n) as c:
        c.set_bodies(pos, np.zeros((n, 3)), mass, np.arange(100, 100 + n, dtype=np.uint64))
        c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        count = c.tree_info()["leaves"]
        want = c.compute_accelerations(0.0, G, 0.0, bh.MODE_PLAIN_FP64)
        acc = c.compute_accelerations(0.0, G, 0.0, mode)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
    # every leaf but the body's own, once
    assert np.all(counts == count - 1)
    err = np.linalg.norm(acc - want, axis=1)
    if mode == bh.MODE_FP64_LIST:
        assert np.all(err <= 1e-13 * np.linalg.norm(want, axis=1))
        return
    # The FP32 forms, per term: coordinates relative to the group off by 2^-22
    # of at most sqrt(3) (three times that of r in r^-3), and the roundings of
    # r^-3 (2^-20) and of a list's partial sum (144 of 2^-24).
    for i in range(0, n, n // 200):
        r = np.linalg.norm(p - p[i], axis=1)
        with np.errstate(divide="ignore", invalid="ignore"):
            term = np.where(r > 0, G * m / (r * r) * (1.3e-6 / r + 1.2e-5), 0.0)
        assert err[i] <= term.sum()
