"""The mesher's scratch: meshes on a device whose memory is nearly taken, and
volumes with more words than the scratch is first made for (which is made
larger and the mesh counted again)."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import cam_params, canon_bits

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _slab(n, seed, z0=300):
    """about n voxels: a wavy surface five voxels thick"""
    side = int((n / 5) ** 0.5)
    z, y, x = np.meshgrid(np.arange(5), np.arange(side), np.arange(side), indexing="ij")
    h = (10 * np.sin(x * 0.05 + seed) + 10 * np.cos(y * 0.07)).astype(np.int64)
    k = (((z0 + h + z) << 20) | ((y % 1024) << 10) | (x % 1024)).ravel()
    d = ((z - 2.1) * 0.01).ravel()
    k, at = np.unique(k, return_index=True)
    return k.astype(np.uint32), np.stack([d[at], np.ones(k.size)], 1).astype(np.float32)


class _LeftFree:
    """The device's memory but `left` bytes, held while inside."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        assert free > self.left + 64 * MB
        self.held = torch.empty(free - self.left, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        import torch
        del self.held
        torch.cuda.empty_cache()


def test_a_mesh_that_fits_is_not_refused(gpu):
    from merge_fusion_gb300 import _lib, kifi
    lib = _lib.load()
    keys, vals = _slab(5_000_000, 1.0)
    more, more_vals = _slab(5_000_000, 1.0, z0=700)

    def volume():
        v = kifi.Volume(1024, 4.0, 0.02, capacity=12_000_000)
        v.insert(keys, vals)
        return v

    def mesh(v):
        nv, ni, pv, pi = C.c_size_t(), C.c_size_t(), C.c_void_p(), C.c_void_p()
        _lib.check(lib.kifi_mesh_device(v.handle, 1, C.byref(nv), C.byref(ni), C.byref(pv), C.byref(pi)))
        return nv.value, ni.value

    a, b = volume(), volume()
    want = kifi.Mesher().Mesh(a, with_indices=True)
    # 5 M voxels: 104 MB of scratch and 59 MB of mesh (the driver keeps some 100 MB)
    with _LeftFree(400 * MB):
        assert mesh(b) == (want[0].shape[0], want[1].size)
        got = kifi.Mesher().Mesh(b, with_indices=True)
    assert np.array_equal(canon_bits(want[0]), canon_bits(got[0])) and np.array_equal(want[1], got[1])
    for v in (a, b):  # the memory is back, the volume larger
        v.insert(more, more_vals)
    want, got = (kifi.Mesher().Mesh(v, with_indices=True) for v in (a, b))
    assert np.array_equal(canon_bits(want[0]), canon_bits(got[0])) and np.array_equal(want[1], got[1])


@pytest.mark.parametrize("bits", [32, 64])
def test_more_words_than_expected(gpu, oracle_cpu, bits):
    # two voxels to a word: 150000 words where the scratch of 300000 voxels first holds 65536
    from merge_fusion_gb300 import kifi
    rng = np.random.default_rng(5)
    z, y, x = np.meshgrid(np.arange(60), np.arange(100), np.arange(0, 800, 32), indexing="ij")
    k = np.stack([(z << 20 | y << 10 | x + i) for i in (4, 5)], -1).ravel().astype(np.uint32)
    vals = np.stack([rng.normal(0, 0.01, k.size), rng.integers(1, 4, k.size)], 1).astype(np.float32)
    v = kifi.Volume(1024, 4.0, 0.02, key_bits=bits)
    v.insert(k, vals)
    ov = oracle_cpu.Volume(1024, 4.0, 0.02)
    ov.keys, ov.values = k, vals
    for wi in (True, False, True):
        got, want = kifi.Mesher().Mesh(v, with_indices=wi), ov.mesh(wi)
        assert np.array_equal(canon_bits(got[0]), canon_bits(want[0])) and want[0].shape[0] > 100000
        assert np.array_equal(got[1], want[1])


def test_a_pipelines_mesh_that_fits_is_not_refused(gpu):
    import torch
    from merge_fusion_gb300 import _lib, scenes
    from merge_fusion_gb300._lib import PipelineDesc, check
    lib = _lib.load()
    seq = scenes.room_scene(n_frames=3, seed=3)
    frames = [torch.from_numpy(np.ascontiguousarray(f).view(np.int16)).cuda() for f in seq.frames]
    torch.cuda.synchronize()

    def run(left):
        d = PipelineDesc()
        d.camera = cam_params(seq.camera).camera()
        d.resolution, d.side_length_m, d.truncation_m = 1024, 4.096, 0.02
        d.icp_iterations, d.mesh_every, d.mesh_with_indices = 0, 1, 1
        d.initial_capacity, d.device = 8 << 20, 0
        pipe = C.c_void_p()
        check(lib.kifi_pipeline_create(C.byref(d), C.byref(pipe)))
        counts = []
        try:
            held = _LeftFree(left)
            held.__enter__()
            try:
                for i in range(3):
                    check(lib.kifi_pipeline_integrate_device(pipe, C.c_void_p(frames[i].data_ptr()), 1,
                                                             seq.world_to_eye_f32(i).ctypes.data_as(C.c_void_p)))
                    nv, ni = C.c_size_t(), C.c_size_t()
                    check(lib.kifi_pipeline_mesh_counts(pipe, C.byref(nv), C.byref(ni)))
                    counts.append((nv.value, ni.value))
            finally:
                held.__exit__()
        finally:
            lib.kifi_pipeline_destroy(pipe)
        return counts

    # the snapshot takes 96 MB, the scratch of the first frame's bound (2.5 M voxels) 50 MB
    assert run(300 * MB) == run(8192 * MB)
