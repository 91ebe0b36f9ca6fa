"""The mesher's row table is cleared whole for every mesh, also where a volume
has fewer runs of voxels than the table needs CTAs: a volume meshed before
with other voxels gives what a new one gives."""
import numpy as np
import pytest

from tests.helpers import canon_bits

pytestmark = pytest.mark.gpu


def _slab(res, b, lo, n, seed):
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(np.arange(4), np.arange(n), np.arange(n), indexing="ij")
    k = (lo[2] + z).astype(np.uint64) << np.uint64(2 * b) | (lo[1] + y).astype(np.uint64) << np.uint64(b) \
        | (lo[0] + x).astype(np.uint64)
    d = 0.01 * (z - 1.5) + rng.normal(0, 0.002, z.shape)
    order = np.argsort(k.ravel())
    return k.ravel()[order], np.stack([d.ravel()[order], np.ones(k.size)], 1).astype(np.float32)


@pytest.mark.parametrize("res,bits", [(512, 32), (1024, 64), (8192, 64)])
@pytest.mark.parametrize("n", [3, 20, 60])
def test_a_second_mesh_equals_a_new_volumes(gpu, res, bits, n):
    from merge_fusion_gb300 import kifi
    used, new = (kifi.Volume(res, 4.0, 0.02, key_bits=bits) for _ in range(2))
    b = 10 if bits == 32 else used.bits_per_axis
    for lo in ((5, 7, 9), (res // 2, res - n - 3, res - 8)):
        k, v = _slab(res, b, lo, n, n)
        k = k.astype(np.uint64 if bits == 64 else np.uint32)
        used.clear()
        used.insert(k, v)
        got = kifi.Mesher().Mesh(used, with_indices=True)
    new.insert(k, v)
    want = kifi.Mesher().Mesh(new, with_indices=True)
    assert got[0].shape[0] > 0 and got[1].shape == want[1].shape
    assert np.array_equal(canon_bits(got[0]), canon_bits(want[0])) and np.array_equal(got[1], want[1])
