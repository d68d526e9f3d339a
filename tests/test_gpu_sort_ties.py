"""The cluster sort where keys share their high halves: runs at the edges of what
a thread, a warp and the passes over the low halves order, in sorted and in
random input, with the keys' low halves distinct and repeated, against numpy's
stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _runs(n, lengths, rng):
    """n keys whose high halves come in runs of the lengths given, in turn."""
    high = np.sort(rng.choice(1 << 31, n, replace=False)).astype(np.uint64)
    start, k = np.zeros(n, np.int64), 0
    i = 0
    while i < n:
        m = lengths[k % len(lengths)]
        start[i:i + m] = i
        i += m
        k += 1
    return high[start] << np.uint64(32)


@pytest.mark.parametrize("n", [300, 1024, 1500, 8191, 16384, 19054, 40001, 65537, 98304])
@pytest.mark.parametrize("lengths", [(16, 1), (17, 1, 1), (31, 32, 33), (64, 2, 65), (255, 1), (256, 3), (257, 1, 1, 1),
                                     (1, 16, 17, 256, 300, 5000), (129, 1, 1, 1, 1, 1, 1, 1)])
@pytest.mark.parametrize("order", ["sorted", "random"])
def test_runs_of_equal_high_halves(bh, n, lengths, order):
    rng = np.random.default_rng(n + len(lengths))
    high = _runs(n, lengths, rng)
    for low in (rng.integers(0, 1 << 32, n, dtype=np.uint64), rng.integers(0, 3, n, dtype=np.uint64)):
        keys = high | low
        keys = np.sort(keys) if order == "sorted" else keys[rng.permutation(n)]
        if order == "sorted":  # a few out of place, as after a step
            for i in rng.integers(0, n - 1, n // 50):
                keys[i], keys[i + 1] = keys[i + 1], keys[i]
        want = np.argsort(keys, kind="stable")
        got, p, _, _, ids = bh.sortBodiesByMortonKey(keys, np.zeros((n, 3)), np.zeros(n), np.zeros((n, 3)),
                                                     np.arange(n, dtype=np.uint64))
        np.testing.assert_array_equal(got, keys[want])
        np.testing.assert_array_equal(ids, want.astype(np.uint64))
