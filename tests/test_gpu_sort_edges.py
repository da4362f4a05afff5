"""The radix sort at the edges of its tiles (2,048 pairs up to 300,000, 4,096
above) and around the window of eight tiles a look-back reads at once: the
stable order by key, ties in input order, against numpy's stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 30, 32])
@pytest.mark.parametrize("n", [2, 31, 2047, 2048, 2049, 8 * 2048, 9 * 2048 + 1, 17 * 2048 - 1, 299_999, 300_000, 300_001,
                               73 * 4096, 82 * 4096 + 1, 700_001])
def test_sort_at_tile_edges(engine, n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[rng.random(n) < 0.3] = keys[0]  # runs of equal keys across tiles
    vals = rng.permutation(n).astype(np.uint32)
    k, v = engine.sort_pairs(keys, vals, bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order])
    assert np.array_equal(v, vals[order])
