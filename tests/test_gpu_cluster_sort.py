"""The sort of small sets in one cluster's shared memory (include/utility.h:23-52):
whole keys and the stable permutation against numpy's stable sort, at the edges
of the block, item and cluster ranges and for each way ties are resolved."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(kind, n, rng):
    hi = rng.integers(0, 1 << 31, n, dtype=np.uint64) << np.uint64(32)
    lo = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    if kind == "random":
        return hi | lo
    if kind == "top_bit":  # all 64 bits take part
        return (hi << np.uint64(1)) | lo
    if kind == "short_ties":  # runs of equal high halves, below and above one block's edge
        return (np.sort(hi)[np.arange(n) // 7 * 7] | (lo & np.uint64(3)))[rng.permutation(n)]
    if kind == "long_ties":  # one high half: every digit decides
        return lo
    if kind == "equal":
        return np.full(n, 0x123456789ABCDEF, np.uint64)
    if kind == "reversed":
        return np.sort(hi | lo)[::-1].copy()
    raise ValueError(kind)


@pytest.mark.parametrize("n", [2, 33, 1023, 1024, 1025, 4097, 8192, 8193, 19054, 24577, 40001, 65535, 65536, 65537,
                               98303, 98304, 98305])
@pytest.mark.parametrize("kind", ["random", "top_bit", "short_ties", "long_ties", "equal", "reversed"])
def test_sort_matches_a_stable_sort(bh, kind, n):
    rng = np.random.default_rng(n)
    keys = _keys(kind, n, rng)
    order = np.argsort(keys, kind="stable")
    pos, vel = rng.random((n, 3)), rng.random((n, 3))
    mass, ids = rng.random(n), np.arange(n, dtype=np.uint64)
    got, p, m, v, ids = bh.sortBodiesByMortonKey(keys, pos, mass, vel, ids)
    np.testing.assert_array_equal(got, keys[order])
    np.testing.assert_array_equal(ids, order.astype(np.uint64))
    np.testing.assert_array_equal(p, pos[order])
    np.testing.assert_array_equal(v, vel[order])
    np.testing.assert_array_equal(m, mass[order])
