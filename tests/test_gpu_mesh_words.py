"""The mesher's words of 32 keys against the oracle: runs across word and row
ends, holes, tile and run edges, operands outside the sign rule's range."""
import numpy as np
import pytest

from tests.helpers import canon_bits

pytestmark = pytest.mark.gpu


def check(kifi, oracle_cpu, keys, vals, bits, wraps=False):
    gv = kifi.Volume(1024, 4.0, 0.02, key_bits=bits)
    gv.insert(keys, vals)
    ov = oracle_cpu.Volume(1024, 4.0, 0.02)
    ov.keys, ov.values = keys, vals
    for wi in (False, True):
        va, ia = kifi.Mesher().Mesh(gv, with_indices=wi)
        vb, ib = ov.mesh(wi)
        assert va.shape == vb.shape, (wi, va.shape, vb.shape)
        assert np.array_equal(canon_bits(va), canon_bits(vb)), wi
        # a cube across the end of a row (x = 1023 and the next row's 0) reads resident voxels like any
        # other, but the reference packs its x + 1 = 1024 into the ids by OR, the mesher by addition
        assert ia.shape == ib.shape
        if not wraps:
            assert np.array_equal(ia, ib), wi


def block(lo, shape, drop, rng):
    """keys of a block at `lo` (x wraps into the next row, as keys do) with a share dropped"""
    z, y, x = np.meshgrid(*(np.arange(s) for s in shape[::-1]), indexing="ij")
    k = ((lo[2] + z).astype(np.int64) << 20) + ((lo[1] + y) << 10) + lo[0] + x
    k = k.ravel()
    k = k[(k >= 0) & (k < 2**30)]
    k = k[rng.random(k.size) >= drop]
    return np.unique(k).astype(np.uint32)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lo", [(28, 3, 3), (60, 1020, 5), (1019, 7, 7), (1000, 1021, 1020), (0, 0, 0)])
@pytest.mark.parametrize("drop", [0.0, 0.05, 0.5])
def test_words_and_rows(gpu, oracle_cpu, bits, lo, drop):
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(7)
    keys = block(lo, (37, 4, 4), drop, rng)
    # zeros, negative and huge operands among ordinary ones
    d = rng.normal(0, 0.01, keys.size)
    w = rng.integers(1, 4, keys.size).astype(float)
    odd = rng.random(keys.size)
    d[odd < 0.02] = 0.0
    d[(odd >= 0.02) & (odd < 0.04)] *= 1e-33
    w[(odd >= 0.04) & (odd < 0.06)] = 0.0
    w[(odd >= 0.06) & (odd < 0.08)] *= -1.0
    w[(odd >= 0.08) & (odd < 0.10)] *= 2.0**31
    wraps = lo[0] + 37 > 1024 or lo[1] + 4 > 1024 or lo[2] + 4 > 1024
    check(kifi, oracle_cpu, keys, np.stack([d, w], 1).astype(np.float32), bits, wraps)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 2047, 2048, 2049, 2081, 19455, 19456, 19457, 70001])
def test_tile_and_run_ends(gpu, oracle_cpu, bits, n):
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(n)
    keys = block((17, 5, 9), (45, 45, 45), 0.1, rng)[:n]
    # a smooth surface and a few flipped signs
    p = np.stack([keys & 1023, keys >> 10 & 1023, keys >> 20], 1).astype(float)
    d = 0.01 * np.sin(p @ np.array([0.31, 0.17, 0.23]))
    d[rng.random(keys.size) < 0.05] *= -1.0
    w = rng.integers(1, 5, keys.size)
    check(kifi, oracle_cpu, keys, np.stack([d, w], 1).astype(np.float32), bits)
