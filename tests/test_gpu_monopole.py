"""The monopole pass's stages (chunks of 512 leaves, then 64 groups per block):
the tree bit for bit against the oracle's at the sizes where a stage is added
or partly filled, and for a system whose nested cells straddle every chunk's
end, which leaves more nodes over than a later stage's block keeps in shared
memory; its second moments against sums over the bodies."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def spread_bits(v):
    out = np.zeros(v.shape, np.uint64)
    for b in range(21):
        out |= ((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return out


def positions_of(keys):
    """Cell centres of 63-bit keys in the unit box."""
    out = np.zeros((len(keys), 3))
    for ax in range(3):
        v = np.zeros(len(keys), np.uint64)
        for b in range(21):
            v |= ((keys >> np.uint64(3 * b + ax)) & np.uint64(1)) << np.uint64(b)
        out[:, ax] = (v.astype(np.float64) + 0.5) / 2.0 ** 21
    return out


def nested_keys(places, seed):
    """`places` groups of 512 keys in cells of depth 3, each holding a chain of
    cells, one inside the other from depth 3 to 20, that ends between its 256th
    and its 257th key: with a first group shifted by half, every 512th key is
    inside all of a chain's cells."""
    rng = np.random.default_rng(seed)
    groups = [np.array([0, (1 << 63) - 1], np.uint64)]  # the box's corners
    for p in range(places):
        base = (p + 1) << 54
        centre = 0
        for d in range(3, 21):
            centre |= int(rng.integers(1, 7)) << (60 - 3 * d)  # room on both sides at every depth
        lower, upper = {base + centre}, {base + centre + 1}
        for d in range(3, 21):
            sh = 60 - 3 * d
            digit = (centre >> sh) & 7
            head = (centre >> (sh + 3)) << (sh + 3)
            below, above = head | ((digit - 1) << sh), head | ((digit + 1) << sh)
            (lower if d % 2 else upper).add(base + (below if d % 2 else above) + int(rng.integers(0, 1 << sh)))
        while len(lower) < 256:
            lower.add(base + int(rng.integers(0, centre)))
        while len(upper) < 256:
            upper.add(base + int(rng.integers(centre + 2, 1 << 54)))
        groups.append(np.array(sorted(lower) + sorted(upper), np.uint64))
    # 255 more at the front put every chunk's end in the middle of a chain
    groups.append(np.arange(1, 256, dtype=np.uint64) << np.uint64(40))
    return np.unique(np.concatenate(groups))


def tree_of(bh, port, pos, mass):
    n = len(mass)
    with bh.Context(n) as c:
        c.set_bodies(pos, np.zeros((n, 3)), mass, np.arange(n, dtype=np.uint64) + np.uint64(100))
        bb = c.compute_bbox(); c.compute_keys(); c.sort_bodies(); c.build_tree(merge=False)
        got = c.export_tree()
        prefix, depth = c.tree_slots()
        spread = c.tree_spread()
        p, _, m, _, _ = c.get_bodies()
    keys = port.keys(p, bb)
    tree = port.tree(keys, p, m, merge=False)
    for a, b, name in zip(got, tree.records(), ("prefix", "depth", "mass", "com")):
        assert_bits_equal(a, b, f"n={n} {name}")
    tree.close()
    return keys, p, m, prefix, depth, spread


@pytest.mark.parametrize("n", [2, 511, 512, 513, 1024, 32767, 32768, 32769, 65537])
def test_tree_at_stage_sizes(bh, port, n):
    pos, _, mass, _ = bh.generate_system(n, max(n, 10), 0.1, 0.05)
    tree_of(bh, port, pos[:n], mass[:n])


def test_nested_cells_at_every_chunk_end(bh, port):
    keys = nested_keys(150, 7)
    rng = np.random.default_rng(8)
    mass = 10.0 ** rng.uniform(12, 20, len(keys))
    sk, p, m, prefix, depth, spread = tree_of(bh, port, positions_of(keys), mass)
    # The straddling cells: more than 384 per 64 chunks.
    cut = np.arange(512, len(sk) - 1, 512)
    common = np.array([20 - (int(a ^ b).bit_length() - 1) // 3 for a, b in zip(sk[cut - 1], sk[cut])])
    assert np.sort(common)[-100:].min() >= 15
    lo = np.searchsorted(sk, prefix, side="left")
    width = np.where(depth == 0, np.uint64(0), np.uint64(1) << (np.uint64(63) - np.uint64(3) * depth.astype(np.uint64)))
    hi = np.where(depth == 0, len(sk), np.searchsorted(sk, prefix + width, side="left"))
    for s in rng.choice(len(prefix), 3000, replace=False):
        w, x = m[lo[s]:hi[s]], p[lo[s]:hi[s]]
        com = (w[:, None] * x).sum(axis=0) / w.sum()
        ref = np.sqrt((w * ((x - com) ** 2).sum(axis=1)).sum() / w.sum())
        assert abs(spread[s] - ref) <= 1e-5 * ref + 1e-12
