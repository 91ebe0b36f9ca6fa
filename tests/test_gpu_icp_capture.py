"""Alignments recorded into a CUDA graph on the caller's stream, as a user's
frame loop does it: against the same alignment enqueued plainly."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import cam_params

pytestmark = pytest.mark.gpu


def _device(frame):
    import torch
    return torch.from_numpy(np.ascontiguousarray(frame).view(np.int16)).cuda()


def _target(icp, d, cam, pose):
    from merge_fusion_gb300._lib import check, load
    check(load().kifi_icp_set_target_from_depth(icp.handle, C.c_void_p(d.data_ptr()), 1, 1,
                                                C.byref(cam_params(cam).camera()), pose.ctypes.data_as(C.c_void_p)))


def _align(icp, d, cam, pose, iterations):
    from merge_fusion_gb300._lib import check, load
    check(load().kifi_icp_align_device(icp.handle, C.c_void_p(d.data_ptr()), 1, C.byref(cam_params(cam).camera()),
                                       pose.ctypes.data_as(C.c_void_p), iterations))


def _capture(stream, fn):
    import torch
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        try:
            fn()
        finally:
            g.capture_end()
    return g


def _rooms(w, h):
    from merge_fusion_gb300 import scenes
    return scenes.room_scene(n_frames=3, seed=6, width=w, height=h, f=585.0 * w / 640.0)


def test_a_frame_larger_than_its_target_needs_no_allocation(gpu):
    import torch
    from merge_fusion_gb300 import kifi
    small, large = _rooms(160, 120), _rooms(320, 240)
    pose = small.eye_to_world_f32(0)
    t, d = _device(small.frames[0]), _device(large.frames[1])
    s = torch.cuda.Stream()
    plain, captured = kifi.ICP(), kifi.ICP(stream=s.cuda_stream)
    torch.cuda.synchronize()
    for icp in (plain, captured):
        _target(icp, t, small.camera, pose)
    _align(plain, d, large.camera, pose, 3)
    g = _capture(s, lambda: _align(captured, d, large.camera, pose, 3))
    with torch.cuda.stream(s):
        g.replay()
    a, b = plain.Result(), captured.Result()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[2], b[2]) and a[2].size == 3


def test_a_graph_searches_the_target_it_finds(gpu, oracle_cpu):
    # captured against a back-projected frame, replayed after the caller put other points there
    import torch
    from merge_fusion_gb300 import kifi
    seq = _rooms(320, 240)
    cam, pose = seq.camera, seq.eye_to_world_f32(0)
    t, d = _device(seq.frames[0]), _device(seq.frames[1])
    s = torch.cuda.Stream()
    icp = kifi.ICP(stream=s.cuda_stream)
    icp.RecordAssociations(True)
    torch.cuda.synchronize()
    _target(icp, t, cam, pose)
    _align(icp, d, cam, pose, 1)  # reserves the records
    torch.cuda.synchronize()
    g = _capture(s, lambda: _align(icp, d, cam, pose, 1))
    target = oracle_cpu.backproject(seq.depth_m(0), cam, pose)
    flat = target.reshape(-1, 3)
    flat[::3] = np.roll(flat[::3], 5, axis=0)  # points that project five pixels' rows from their own
    icp.SetTarget(target, pose)
    with torch.cuda.stream(s):
        g.replay()
    torch.cuda.synchronize()
    gi, gl = icp.Associations()
    oi, ol = oracle_cpu.icp_associate(seq.depth_m(1), cam, pose, target, pose)
    assert np.array_equal(gi, oi) and np.array_equal(gl.view(np.uint32), ol.view(np.uint32))
