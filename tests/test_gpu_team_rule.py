"""The masked walks on both sides of the lines where the warps to a group change
above theta 1.3: from teams of 4 to one warp at 320 (theta / 1.3)^-2 bodies to an
SM (list), 576 (theta / 1.3)^-4 (group) and 1,344 (theta / 1.3)^-4 (FP32), with
152 SMs, and from teams of 8 to 4 at 128 (64 in the list form).  The list form's
counts are the oracle's; at a line the FP32 forms with a team and with one warp
meet the same nodes, so their mean counts differ by the last body's at most."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import G

pytestmark = pytest.mark.gpu


def forces(bh, n, theta, mode, extra=0):
    pos, vel, mass, ids = bh.generate_system(11, n + extra, 0.1, 0.05)
    pos, vel, mass, ids = pos[:n], vel[:n], mass[:n], ids[:n]
    with bh.Context(n) as c:
        c.set_bodies(pos, vel, mass, ids)
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree()
        acc = c.compute_accelerations(theta, G, 0.0, mode)
        counts = c.interaction_counts()
        p, _, m, _, _ = c.get_bodies()
        sample = np.unique(np.linspace(0, n - 1, 256).astype(np.int64))
        want = c.direct_sum(sample, G)
    return bb, p, m, acc, counts, sample, want


@pytest.mark.parametrize("n,theta", [(20550, 2.0), (20551, 2.0), (48640, 1.3), (48641, 1.3), (9728, 1.3), (9729, 1.3)])
def test_list(bh, port, n, theta):
    bb, p, m, acc, counts, _, _ = forces(bh, n, theta, bh.MODE_FP64_LIST)
    keys = port.keys(p, bb)
    want, cnt = port.accelerations(port.tree(keys, p, m), keys, p, theta, G, 0.0, bb, count=True)
    assert np.array_equal(counts, cnt)
    assert np.all(np.linalg.norm(acc - want, axis=1) <= 1e-13 * np.linalg.norm(want, axis=1))


@pytest.mark.parametrize("line,theta,mode", [(19456, 2.0, "group"), (19456, 1.3, "group"), (38155, 1.6, "group"),
                                             (19456, 1.3, "far"), (36466, 2.0, "far"), (89029, 1.6, "far")])
def test_fp32(bh, line, theta, mode):
    mode = {"far": bh.MODE_FP32_FAR, "group": bh.MODE_FP32_GROUP}[mode]
    mean = []
    for n in (line, line + 1):
        _, _, _, acc, counts, sample, want = forces(bh, n, theta, mode, line + 1 - n)
        err = np.linalg.norm(acc[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert np.median(err) < 1e-5 and np.all(err < 1e-2)
        mean.append(counts.mean())
    assert abs(mean[1] / mean[0] - 1) < 1e-2
