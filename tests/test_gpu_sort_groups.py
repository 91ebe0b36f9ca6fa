"""Sorts at the edges of the look-back's tiles (2048 keys) and groups of 16
tiles, with a CTA per tile and with tiles from the counter, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047, 2049, 15 * 2048, 16 * 2048, 16 * 2048 + 1, 17 * 2048, 32 * 2048 - 1,
                               33 * 2048 + 5, 608 * 2048, 609 * 2048, 700 * 2048 + 3])
def test_sort_at_group_edges(gpu, n):
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    keys[: n // 3] &= 0xffff  # uneven digits
    vals = np.arange(n, dtype=np.uint32)
    order = np.argsort(keys, kind="stable")
    k, v = kifi.radix_sort(keys, vals)
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])
