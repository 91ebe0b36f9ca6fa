"""A target that does not fit the device's memory is refused; the context's next
target is used.  Until then it has none, and aligning says so."""
import numpy as np
import pytest

from tests.helpers import cam_params
from tests.test_gpu_mesh_memory import MB, _LeftFree

pytestmark = pytest.mark.gpu


def _room(oracle_cpu):
    from merge_fusion_gb300 import scenes
    seq = scenes.room_scene(n_frames=2, seed=6, width=160, height=120, f=146.25)
    pose = seq.eye_to_world_f32(0)
    return seq, pose, oracle_cpu.backproject(seq.depth_m(0), seq.camera, pose)


def _refuse(icp, pose):
    from merge_fusion_gb300 import _lib
    large = np.ones((5000, 6000, 3), np.float32)  # 550 MB on the device
    with _LeftFree(300 * MB):
        with pytest.raises(_lib.KifiError) as err:
            icp.SetTarget(large, pose)
    assert err.value.status == _lib.KIFI_ERR_OUT_OF_MEMORY


def test_the_next_target_is_used(gpu, oracle_cpu):
    from merge_fusion_gb300 import kifi
    seq, pose, target = _room(oracle_cpu)
    icp = kifi.ICP()
    icp.SetTarget(target, pose)
    want = icp.AlignToTarget(seq.depth_m(1), pose, cam_params(seq.camera), 2)
    _refuse(icp, pose)
    icp.SetTarget(target, pose)
    assert np.array_equal(icp.AlignToTarget(seq.depth_m(1), pose, cam_params(seq.camera), 2), want)


def test_a_refused_target_leaves_none(gpu, oracle_cpu):
    from merge_fusion_gb300 import _lib, kifi
    seq, pose, target = _room(oracle_cpu)
    icp = kifi.ICP()
    icp.SetTarget(target, pose)
    _refuse(icp, pose)
    with pytest.raises(_lib.KifiError) as err:
        icp.AlignToTarget(seq.depth_m(1), pose, cam_params(seq.camera), 2)
    assert err.value.status == _lib.KIFI_ERR_INVALID_ARGUMENT
