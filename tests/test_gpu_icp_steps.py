"""The association of an alignment's later steps, pair for pair and len^2 bit
for bit, against the oracle's full 21x21 scan at the pose that the steps before
have reached: what a step reads is decided by what the last one left (winners,
regions staged ahead, each tile's way to search), in every shape of launch --
no more tiles than SMs, up to two per SM, more, targets finer than the frame,
targets that must be searched whole -- and with few steps and many.  One context
for targets of changing size, as a program keeps it."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import cam_params, posed

pytestmark = pytest.mark.gpu


def _room(w, h):
    from merge_fusion_gb300 import scenes
    return scenes.room_scene(n_frames=4, seed=8, width=w, height=h, f=585.0 * w / 640.0)


def _check(icp, oracle_cpu, seq, i, guess, target, synth_e2w, steps, cam=None):
    cam, depth = cam or seq.camera, seq.depth_m(i)
    found = 0
    for n in steps:
        icp.RecordAssociations(False)
        pose = icp.AlignToTarget(depth, guess, cam_params(cam), n - 1) if n > 1 else guess
        icp.RecordAssociations(True)
        icp.AlignToTarget(depth, guess, cam_params(cam), n)
        gi, gl = icp.Associations()
        oi, ol = oracle_cpu.icp_associate(depth, cam, pose, target, synth_e2w)
        bad = np.nonzero(gi != oi)[0]
        assert bad.size == 0, (n, bad.size, bad[:5], gi[bad[:5]], oi[bad[:5]])
        assert np.array_equal(gl.view(np.uint32), ol.view(np.uint32)), n
        found += int((gi >= 0).sum())
    return found


STEPS = (2, 3, 5, 9, 15)


def test_depth_targets(gpu, oracle_cpu):
    from merge_fusion_gb300 import kifi
    icp = kifi.ICP()
    for w, h in ((640, 480), (320, 240), (1024, 848), (97, 61), (515, 421)):
        seq = _room(w, h)
        prev = seq.eye_to_world_f32(0)
        target = oracle_cpu.backproject(seq.depth_m(0), seq.camera, prev)
        icp.SetTargetFromDepth(seq.frames[0], cam_params(seq.camera), prev)
        for i, off in ((1, (0.0, 0.0, 0.0)), (3, (0.02, -0.01, 0.01)), (2, (-0.08, 0.05, 0.1))):
            n = _check(icp, oracle_cpu, seq, i, posed(prev, off), target, prev, STEPS if w < 1000 else (3, 6))
            assert n > w * h // 40


@pytest.mark.parametrize("kind", ["points", "scattered", "offcentre"])
def test_measured_targets(gpu, oracle_cpu, kind):
    from merge_fusion_gb300 import kifi
    icp = kifi.ICP()
    for w, h in ((320, 240), (640, 480)):
        seq = _room(w, h)
        cam = list(seq.camera)
        if kind == "offcentre":  # (EyeToClipRH shifts the image by (W - 2 cx) W / 2 pixels: five and ten)
            cam[4] += 1.0 / 64
        prev = seq.eye_to_world_f32(0)
        target = oracle_cpu.backproject(seq.depth_m(0), cam, prev)
        if kind == "scattered":  # every third pixel's point belongs to another pixel
            flat = target.reshape(-1, 3)
            flat[::3] = np.roll(flat[::3], 5, axis=0)
        icp.SetTarget(target, prev)
        for i in (1, 3):
            _check(icp, oracle_cpu, seq, i, prev, target, prev, (2, 5, 9, 12), cam)


def test_fine_targets(gpu, oracle_cpu):
    import torch
    from merge_fusion_gb300 import _lib, kifi
    seq = _room(640, 480)
    prev = seq.eye_to_world_f32(0)
    cloud = oracle_cpu.backproject(seq.depth_m(0), seq.camera, prev).reshape(-1, 3)
    cloud = np.ascontiguousarray(cloud[np.any(cloud != 0, axis=1)], np.float32)
    pts = torch.from_numpy(cloud).cuda()
    torch.cuda.synchronize()
    w2c = oracle_cpu.mat_mul(oracle_cpu.eye_to_clip(seq.camera), oracle_cpu.invert_transform(prev))
    icp = kifi.ICP()
    _lib.check(_lib.load().kifi_icp_set_target_bin_device(icp.handle, C.c_void_p(pts.data_ptr()), cloud.shape[0],
                                                          w2c.ctypes.data_as(C.c_void_p), 1024, 768,
                                                          prev.ctypes.data_as(C.c_void_p)))
    target = oracle_cpu.bin_points(cloud, w2c, 1024, 768)
    for i in (1, 3):
        _check(icp, oracle_cpu, seq, i, prev, target, prev, (1, 2, 4, 9))
