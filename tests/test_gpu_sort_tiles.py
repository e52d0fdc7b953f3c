"""The radix sort at the edges of its tiles: the small and the large tile, the
counts at which a scatter block adds the histograms up itself (160 tiles of 1,024
keys) and at which the large tile takes over (2^20 keys); stable, so that equal
keys keep their order."""

import numpy as np
import pytest

import molla_b200 as m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [7, 18])
@pytest.mark.parametrize("n", [1, 255, 1023, 1024, 1025, 160 * 1024, 160 * 1024 + 1, 1 << 20, (1 << 20) + 1])
def test_sort_at_tile_edges(engine, n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, size=n, dtype=np.uint64).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    k, v = m.radix_sort_pairs(engine, keys, vals, bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])
