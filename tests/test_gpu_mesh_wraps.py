"""Triangle indices of blocks that cross the ends of key rows, compared whole.
The reference packs the x + 1 = 1024 of a cube across a row's end into an id by
OR; the mesher adds, so the oracle's indices differ there.  Here a host mesher
that forms ids by addition stands beside it: on blocks within their rows it gives
the oracle's indices."""
import os
import re

import numpy as np
import pytest

from tests.helpers import canon_bits
from tests.test_gpu_mesh_words import block

pytestmark = pytest.mark.gpu

_CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "merge_fusion_gb300", "csrc")
_TABLE = [int(w, 16) for w in re.findall(r"0x([0-9a-f]{16})ull", open(os.path.join(_CSRC, "mc_table.cuh")).read())]
_CORNER = [4, 0, 0, 1, 6, 2, 2, 3, 5, 4, 0, 1]  # per edge (Mesher.cpp:206-218)
_AXIS = [0, 2, 0, 2, 0, 2, 0, 2, 1, 1, 1, 1]
_BIT = [2, 3, 6, 7, 1, 0, 5, 4]  # the case bit of each corner (:191-199)


def host_indices(keys, vals):
    """Mesher.cpp:85-229 and :25-44 in Python: the indices of Mesh(verts, indices)."""
    n = keys.size
    at = {int(k): i for i, k in enumerate(keys)}
    with np.errstate(all="ignore"):
        d = vals[:, 0] / vals[:, 1]
        product = lambda i, j: d[i] * d[j]  # noqa: E731
        delta = [(c & 1) + ((c >> 1 & 1) << 10) + ((c >> 2) << 20) for c in range(8)]
        ids, tris = [], []
        for i in range(n - 2, -1, -1):
            if vals[i, 1] == 0.0:
                continue
            k = int(keys[i])
            for axis in range(3):
                j = at.get(k + delta[1 << axis])
                if j is None or (axis and j == n - 1):  # the +y and +z pointers end at n - 2
                    continue
                if vals[j, 1] > 0.0 and product(i, j) <= 0.0:
                    ids.append(3 * k + axis)
            corners = [at.get(k + q) for q in delta]
            if any(j is None or vals[j, 1] == 0.0 for j in corners) or any(corners[c] == n - 1 for c in (0, 2, 4, 6)):
                continue
            word = _TABLE[sum(1 << _BIT[c] for c in range(8) if d[corners[c]] < 0.0)]
            for t in range(3 * (word >> 60)):
                e = word >> (4 * t) & 15
                tris.append(3 * (k + delta[_CORNER[e]]) + _AXIS[e])
    ids, tris = np.sort(np.array(ids, np.int64)), np.array(tris, np.int64)
    missing = tris[~np.isin(tris, ids)]
    bound = missing.min() if missing.size else np.int64(2**62)
    return np.where(tris < bound, np.searchsorted(ids, tris), tris).astype(np.uint32)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lo", [(28, 3, 3), (60, 1020, 5), (1019, 7, 7), (1000, 1021, 1020), (1005, 2, 1022), (987, 1023, 0)])
@pytest.mark.parametrize("drop", [0.0, 0.05, 0.3])
def test_indices_by_addition(gpu, oracle_cpu, bits, lo, drop):
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(11)
    keys = block(lo, (37, 5, 4), drop, rng)
    w = rng.integers(1, 4, keys.size).astype(float)
    odd = rng.random(keys.size)
    d = rng.normal(0, 0.01, keys.size)
    # no missing vertices, and some (weights of zero and below), by the drop
    if drop == 0.05:
        w[odd < 0.01] *= -1.0
    vals = np.stack([d, w], 1).astype(np.float32)
    gv = kifi.Volume(1024, 4.0, 0.02, key_bits=bits)
    gv.insert(keys, vals)
    v, i = kifi.Mesher().Mesh(gv, with_indices=True)
    want = host_indices(keys, vals)
    assert i.size and np.array_equal(i, want)
    ov = oracle_cpu.Volume(1024, 4.0, 0.02)
    ov.keys, ov.values = keys, vals
    vb, ib = ov.mesh(True)
    assert np.array_equal(canon_bits(v), canon_bits(vb))
    if lo[0] + 37 <= 1024 and lo[1] + 5 <= 1024 and lo[2] + 4 <= 1024:
        assert np.array_equal(ib, want)
