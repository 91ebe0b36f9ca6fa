"""Merges whose tiles start at any offset of the resident keys and hold none,
a few, up to 256 and more new keys, against a host merge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("resident", [0, 1, 1023, 2049, 20011])
@pytest.mark.parametrize("new", [1, 3, 255, 256, 257, 2500])
@pytest.mark.parametrize("spread", [False, True])
def test_insert_equals_host_merge(gpu, bits, resident, new, spread):
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(resident + new)
    pool = np.sort(rng.choice(2**30, resident + 3 * new, replace=False).astype(np.uint32))
    # new keys scattered among the resident ones, or side by side from the middle on
    pick = np.zeros(pool.size, bool)
    if spread:
        pick[rng.choice(pool.size, new, replace=False)] = True
    else:
        lo = (pool.size - new) // 2
        pick[lo:lo + new] = True
    a, b = pool[~pick], pool[pick]
    va = rng.random((a.size, 2), np.float32)
    vb = rng.random((b.size, 2), np.float32)
    v = kifi.Volume(1024, 4.0, 0.02, key_bits=bits)
    v.insert(a, va)
    v.insert(b, vb)
    k, x = v.export()
    order = np.argsort(np.concatenate([a, b]), kind="stable")
    assert np.array_equal(k, np.concatenate([a, b])[order])
    assert np.array_equal(x, np.concatenate([va, vb])[order])
