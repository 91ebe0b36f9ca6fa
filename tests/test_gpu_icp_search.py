"""The association's pruned window search against the oracle's full 21x21
scan, pair for pair and len^2 bit for bit, over the forms of target it tells
apart: a back-projected frame aligned with its own camera, a cloud binned
through the aligning matrix, points of the caller's (measured), and the ones
that must be searched whole -- scattered points, a principal point off the
centre, a pose that is not rigid, sources close to the eye."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import cam_params, posed

pytestmark = pytest.mark.gpu


def _pairs(icp):
    i, l2 = icp.Associations()
    return i, l2.view(np.uint32)


def _frames(w, h, seed=6, scale=1.0):
    from merge_fusion_gb300 import scenes
    return scenes.room_scene(n_frames=4, seed=seed, width=w, height=h, f=585.0 * w / 640.0, scale=scale)


def _check(icp, oracle_cpu, depth, cam, guess, target, synth_e2w):
    icp.RecordAssociations(True)
    icp.AlignToTarget(depth, guess, cam_params(cam), 1)
    gi, gl = _pairs(icp)
    oi, ol = oracle_cpu.icp_associate(depth, cam, guess, target, synth_e2w)
    bad = np.nonzero(gi != oi)[0]
    assert bad.size == 0, (bad.size, bad[:5], gi[bad[:5]], oi[bad[:5]])
    assert np.array_equal(gl, ol.view(np.uint32))
    return int((gi >= 0).sum())


@pytest.mark.parametrize("w,h", [(640, 480), (320, 240), (515, 421), (97, 61), (724, 543), (12, 9)])
@pytest.mark.parametrize("kind", ["depth", "points", "scattered"])
def test_search_equals_full_scan(gpu, oracle_cpu, kind, w, h):
    from merge_fusion_gb300 import kifi
    seq = _frames(w, h)
    cam, prev = seq.camera, seq.eye_to_world_f32(0)
    target = oracle_cpu.backproject(seq.depth_m(0), cam, prev)
    icp = kifi.ICP()
    if kind == "depth":
        icp.SetTargetFromDepth(seq.frames[0], cam_params(cam), prev)
    else:
        if kind == "scattered":  # every third pixel's point belongs to another pixel
            flat = target.reshape(-1, 3)
            flat[::3] = np.roll(flat[::3], 5, axis=0)
        icp.SetTarget(target, prev)
    for i, off in ((1, (0.0, 0.0, 0.0)), (3, (0.01, -0.006, 0.004)), (2, (-0.09, 0.05, 0.2)), (0, (0.0, 0.0, 0.0))):
        n = _check(icp, oracle_cpu, seq.depth_m(i), cam, posed(prev, off), target, prev)
        assert n > w * h // 400 or w < 97


@pytest.mark.parametrize("w,h", [(1024, 768), (640, 480), (333, 250)])
def test_search_on_binned_clouds(gpu, oracle_cpu, w, h):
    import torch
    from merge_fusion_gb300 import _lib, kifi
    from merge_fusion_gb300._lib import check
    seq = _frames(640, 480)
    cam, prev = seq.camera, seq.eye_to_world_f32(0)
    cloud = oracle_cpu.backproject(seq.depth_m(0), cam, prev).reshape(-1, 3)
    cloud = np.ascontiguousarray(cloud[np.any(cloud != 0, axis=1)], np.float32)
    pts = torch.from_numpy(cloud).cuda()
    torch.cuda.synchronize()
    icp = kifi.ICP()
    lib, w2e = _lib.load(), oracle_cpu.invert_transform(prev)
    other = posed(prev, (0.02, 0.01, -0.03))
    # binned through the aligning matrix, and through another one (measured)
    for bin_pose in (prev, other):
        w2c = oracle_cpu.mat_mul(oracle_cpu.eye_to_clip(cam), oracle_cpu.invert_transform(bin_pose))
        target = oracle_cpu.bin_points(cloud, w2c, w, h)
        check(lib.kifi_icp_set_target_bin_device(icp.handle, C.c_void_p(pts.data_ptr()), cloud.shape[0],
                                                 w2c.ctypes.data_as(C.c_void_p), w, h,
                                                 prev.ctypes.data_as(C.c_void_p)))
        for off in ((0.0, 0.0, 0.0), (0.015, -0.01, 0.02)):
            _check(icp, oracle_cpu, seq.depth_m(1), cam, posed(prev, off), target, prev)


@pytest.mark.parametrize("form", ["offcentre", "offcentre_little", "scaled_pose", "near", "other_camera", "empty"])
def test_search_where_geometry_does_not_hold(gpu, oracle_cpu, form):
    from merge_fusion_gb300 import kifi
    seq = _frames(320, 240)
    cam, prev = list(seq.camera), seq.eye_to_world_f32(0).copy()
    depth0, depth1 = seq.depth_m(0).copy(), seq.depth_m(1).copy()
    # (EyeToClipRH shifts the image by (W - 2 cx) W / 2 pixels: 80 and 5 of them)
    if form == "offcentre":
        cam[4] += 0.25
    if form == "offcentre_little":
        cam[4] += 1.0 / 64
    if form == "scaled_pose":
        prev[:12] *= np.float32(1.02)
    if form == "near":
        depth0 *= np.float32(0.05)
        depth1 *= np.float32(0.05)
    if form == "empty":
        depth0[:] = 0
    target = oracle_cpu.backproject(depth0, cam, prev)
    icp = kifi.ICP()
    icp.SetTargetFromDepth(depth0, cam_params(cam), prev)
    if form == "other_camera":  # the aligning camera is not the one that took the target
        cam[2] *= 1.01
        cam[3] *= 0.99
    for off in ((0.0, 0.0, 0.0), (0.01, 0.005, -0.02)):
        n = _check(icp, oracle_cpu, depth1, cam, posed(prev, off), target, prev)
        assert (n == 0) == (form in ("empty", "offcentre"))
