"""Workloads of the fusion path, as a user's program runs them through the
package's public entry points: fusing depth frames into a volume and meshing
it, aligning a frame by ICP, the tracking pipelines (open loop fed from the
host or from the device, and the reference's closed loop), a batch of uneven
sequences, and the learned pose proposer's forward and backward passes.

A case is a plain dict; ``prepare`` builds what the program holds before the
call (frames on the GPU or on the host, a volume that already holds part of
a room, the network's weights), ``run`` is one pass, ``work`` the bytes and
operations such a pass cannot do without and ``exact`` the same result in
64 bits where the path computes numbers that have one."""
import ctypes as C
import math
import os

import numpy as np
import torch

import merge_fusion_gb300
from merge_fusion_gb300 import _lib, kifi, proposer, scenes
from merge_fusion_gb300._lib import Camera, PipelineDesc, check

WEIGHTS = os.path.join(os.path.dirname(merge_fusion_gb300.__file__), "weights", "proposer_room.npz")
F_PER_W = 585.0 / 640.0  # focal length in pixels per pixel of width of the room's camera


# ------------------------------------------------------------------- cases

def listed():
    return [
        # ICP::Align exactly as the reference's callers use it: a host frame against a host
        # point buffer, its four iterations; the smallest call, made of launches and latency.
        {"name": "icp_points_320x240_4it", "kind": "icp", "form": "points", "width": 320, "height": 240,
         "iterations": 4, "step": 1},
        # Tracking one frame against the one before, both on the device, to convergence.
        {"name": "icp_depth_640x480_15it", "kind": "icp", "form": "depth", "width": 640, "height": 480,
         "iterations": 15, "step": 1},
        # The small scan: ten 320x240 frames of the sphere scene into an empty 8 mm volume, read back.
        {"name": "scan_320x240_8mm", "kind": "scan", "scene": "sphere", "width": 320, "height": 240, "frames": 10,
         "res": 512, "voxel_mm": 8, "stride": 1, "out": "export"},
        # A Kinect-size scan of a quarter of a room at 4 mm (every third frame) from an empty volume, then its mesh.
        {"name": "scan_640x480_4mm", "kind": "scan", "scene": "room", "width": 640, "height": 480, "frames": 30,
         "res": 1024, "voxel_mm": 4, "stride": 3, "out": "mesh"},
        # The fine volume with 64-bit keys: 512x424 frames at 2 mm, then the vertices-only mesh.
        {"name": "scan_512x424_2mm_key64", "kind": "scan", "scene": "room", "width": 512, "height": 424,
         "frames": 10, "res": 2048, "voxel_mm": 2, "stride": 1, "out": "verts"},
        # Meshing a room-size model: 36 frames all around a 4 mm room.
        {"name": "mesh_room_4mm", "kind": "mesh", "width": 640, "height": 480, "res": 1024, "voxel_mm": 4,
         "warm": 36, "indices": True},
        # The headline: live frames from page-locked host memory, fused into a mapped room and
        # tracked with 15 iterations each, a mesh every ten frames, every frame's pose read back.
        {"name": "track_host_640x480_4mm", "kind": "track", "feed": "host", "width": 640, "height": 480,
         "res": 1024, "voxel_mm": 4, "frames": 10, "iterations": 15, "mesh_every": 10, "warm": 30},
        # The same pipeline on the largest frames, already on the device, queued without waiting.
        {"name": "track_device_1024x848_4mm", "kind": "track", "feed": "device", "width": 1024, "height": 848,
         "res": 1024, "voxel_mm": 4, "frames": 10, "iterations": 15, "mesh_every": 0, "warm": 30},
        # The reference's own tracking loop: align against the model's binned mesh, fuse, mesh, bin.
        {"name": "closed_loop_640x480_8mm", "kind": "closed", "width": 640, "height": 480, "res": 512,
         "voxel_mm": 8, "frames": 5, "iterations": 4, "warm": 0},
        # Eight independent sequences of uneven sizes stepped together.
        {"name": "batch_8_mixed", "kind": "batch", "scenes": 8, "spec_seed": 7, "steps": 4, "iterations": 15},
        # The warm start of one alignment: one frame pair to a network input, one padded batch of 8.
        {"name": "propose_pair_batch8", "kind": "predict", "batch": 8, "pairs": 1},
        # One training batch, forward and backward.
        {"name": "propose_gradients_batch256", "kind": "gradients", "batch": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["icp", "icp", "scan", "scan", "mesh", "track", "track", "closed", "batch", "predict",
                       "gradients"])
    # frame sizes from 320x240 to 1024x848 and odd ones between (multiples of 4 wide, as kifi asks)
    w = 4 * rng.randint(80, 256)
    h = int(w * rng.choice([0.75, 0.828125])) - rng.randint(0, 3)
    if kind == "icp":
        return {"kind": "icp", "form": rng.choice(["points", "depth", "depth"]), "width": w - rng.randint(0, 3),
                "height": h, "iterations": rng.randint(2, 20), "step": rng.randint(1, 3)}
    res, vox = rng.choice([(512, 8), (1024, 4), (1024, 4), (2048, 2)])
    if kind == "scan":
        return {"kind": "scan", "scene": "room", "width": w, "height": h, "frames": rng.randint(3, 20), "res": res,
                "voxel_mm": vox, "stride": rng.randint(1, 3), "out": rng.choice(["mesh", "verts", "export"])}
    if kind == "mesh":
        return {"kind": "mesh", "width": w, "height": h, "res": res, "voxel_mm": vox,
                "warm": rng.randint(1, 36 if vox > 2 else 8), "indices": rng.random() < 0.7}
    if kind == "track":
        return {"kind": "track", "feed": rng.choice(["host", "device"]), "width": w, "height": h, "res": res,
                "voxel_mm": vox, "frames": rng.randint(3, 10 if vox > 2 else 5), "iterations": rng.randint(4, 15),
                "mesh_every": rng.choice([0, 5, 10]), "warm": rng.randint(0, 30 if vox > 2 else 6)}
    if kind == "closed":
        return {"kind": "closed", "width": w, "height": h, "res": 512, "voxel_mm": 8,
                "frames": rng.randint(2, 5), "iterations": rng.randint(2, 6), "warm": 0}
    if kind == "batch":
        most = next(work(c) for c in listed() if c["kind"] == "batch")
        while True:
            c = {"kind": "batch", "scenes": rng.randint(2, 8), "spec_seed": rng.randint(0, 999),
                 "steps": rng.randint(1, 4), "iterations": rng.randint(4, 15)}
            if all(work(c)[k] <= most[k] for k in most):
                return c
    b = 8 * _log_int(rng, 1, 32)
    if kind == "predict":
        return {"kind": "predict", "batch": b, "pairs": rng.choice([1, b])}
    return {"kind": "gradients", "batch": b}


# ------------------------------------------------------------------ inputs

def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


class _Owned:
    """A C handle and the call that frees it."""

    def __init__(self, handle, free):
        self.h, self._free = handle, free

    def __del__(self):
        if self.h is not None:
            self._free(self.h)
            self.h = None


class _DeviceView:
    def __init__(self, address, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (address, False),
                                         "version": 2, "strides": None}


def _view(address, shape, typestr, dtype):
    """Device memory of the library as a tensor, without a copy."""
    if not address or 0 in shape:
        return torch.empty(shape, dtype=dtype, device="cuda")
    return torch.as_tensor(_DeviceView(address, shape, typestr), device="cuda")


def _seed(seed):
    return int(seed) % 1000003


def _params(w, h):
    f = F_PER_W * w
    return kifi.DepthSensorParams((w, h), (f, f), (w / 2.0, h / 2.0), (0.4, 4.0))


def _camera(w, h):
    return _params(w, h).camera()


def _room(seed, w, h, numbers):
    """Depth frames (n, h, w) of the seeded room, uint16 millimetres as an
    int16 bit pattern on the device, at these places of its trajectory, and
    their eye-to-world poses."""
    frames, poses, k = [], [], 0
    while k < len(numbers):  # runs of consecutive numbers are rendered together
        n = 1
        while k + n < len(numbers) and numbers[k + n] == numbers[k] + n:
            n += 1
        fr, ps = scenes.render_room_torch(n, seed=_seed(seed), width=w, height=h, f=F_PER_W * w,
                                          first_frame=numbers[k], device="cuda", chunk=1 << 18, noise="device")
        frames.append(fr)
        poses += ps
        k += n
    return torch.cat(frames), poses


def _w2e(poses):
    return np.stack([scenes.kifi_matrix(np.linalg.inv(p)) for p in poses])


def _warm_numbers(n):
    """n places spread over one turn of the trajectory (one degree a frame)."""
    return [int(round(360.0 * k / n)) for k in range(n)]


def _back_and_forth(n):
    return list(range(n)) + list(range(n - 2, 0, -1))


def _host_u16(frames):
    """The frames in page-locked host memory."""
    out = torch.empty(frames.shape, dtype=torch.int16, pin_memory=True)
    out.copy_(frames)
    return out


# an upper bound of the voxels a room or its scan holds, per frame size and voxel size
def _capacity(c, frames):
    px = c["width"] * c["height"]
    room = {8: 6 << 20, 4: 24 << 20, 2: 96 << 20}[c["voxel_mm"]]
    return min(8 * px * frames, room) + 8 * px * (c.get("frames", 1) + 4)


def _side(c):
    return c["res"] * c["voxel_mm"] * 1e-3


def _trunc(c):
    return (6 if c.get("scene") == "sphere" or c["voxel_mm"] == 8 else 5) * 0.5e-3 * c["voxel_mm"] * 2


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


# --------------------------------------------------------------------- ICP

def _prepare_icp(c, seed):
    w, h = c["width"], c["height"]
    frames, poses = _room(seed, w, h, [40, 40 + c["step"]])
    prev = scenes.kifi_matrix(poses[0])
    s = {"kind": "icp", "c": c, "icp": kifi.ICP(), "params": _params(w, h), "guess": prev, "frames": frames}
    if c["form"] == "points":
        s["points"] = _backproject(frames[0], _params(w, h), prev, torch.float32).cpu().numpy()
        s["raw"] = (frames[1].to(torch.int32) & 0xFFFF).to(torch.float32).mul_(0.001).cpu().numpy()
    return s


def _run_icp(s):
    c, icp = s["c"], s["icp"]
    if c["form"] == "points":
        pose = icp.Align(s["raw"], s["guess"], s["points"], s["guess"], s["params"], iterations=c["iterations"])
    else:
        lib, cam = _lib.load(), s["params"].camera()
        check(lib.kifi_icp_set_target_from_depth(icp.handle, C.c_void_p(s["frames"][0].data_ptr()), 1, 1,
                                                 C.byref(cam), _ptr(s["guess"])))
        check(lib.kifi_icp_align_device(icp.handle, C.c_void_p(s["frames"][1].data_ptr()), 1, C.byref(cam),
                                        _ptr(s["guess"]), c["iterations"]))
        pose = None
    single, double, pairs, rms = icp.Result()
    return {"pose": single if pose is None else pose, "pose64": double, "pairs": pairs, "rms": rms}


def _backproject(frame, params, pose16, dtype):
    """World points (h, w, 3) of a depth frame; (0, 0, 0) where it has none."""
    (w, h), (fx, fy), (cx, cy) = params.resolution, params.focal_length, params.principal_point
    d = (frame.to(torch.int32) & 0xFFFF).to(dtype) * 0.001
    u = torch.arange(w, device=d.device, dtype=dtype)
    v = torch.arange(h, device=d.device, dtype=dtype)[:, None]
    eye = torch.stack([(u + 0.5 - cx) / fx * d, (cy - 0.5 - v) / fy * d, -d, torch.ones_like(d)], -1)
    m = torch.tensor(np.asarray(pose16).reshape(4, 4).T.copy(), device=d.device, dtype=dtype)
    p = (eye @ m.T)[..., :3]
    return torch.where(d[..., None] > 0, p, torch.zeros_like(p))


def _exact_icp(c, seed):
    """The reference's AlignStep (21x21 window around each source's projection,
    every row and fourth column, nearest point within 10 cm, Horn's closed
    form) in float64."""
    s = _prepare_icp(c, seed)
    prm = s["params"]
    (w, h), (fx, fy), (cx, cy) = prm.resolution, prm.focal_length, prm.principal_point
    f64, dev = torch.float64, "cuda"
    guess = np.asarray(s["guess"], np.float64).reshape(4, 4).T
    if c["form"] == "points":
        target = torch.from_numpy(s["points"]).to(dev).to(f64)
        d = torch.from_numpy(s["raw"]).to(dev).to(f64)
    else:
        target = _backproject(s["frames"][0], prm, s["guess"], f64)
        d = (s["frames"][1].to(torch.int32) & 0xFFFF).to(f64) * 0.001
    d = d[:, ::4]
    ok = d != 0
    v0, u0 = torch.nonzero(ok, as_tuple=True)
    d = d[ok]
    # the source's eye point, with the half-pixel offsets of the reference
    eye = torch.stack([(u0 * 4 + 0.5 - cx) / fx * d, (cy - 0.5 - v0) / fy * d, -d, torch.ones_like(d)], -1)
    zn, zf = prm.sensible_range
    clip = np.array([[2 * fx / w, 0, 0, 0], [0, 2 * fy / h, 0, 0], [0, 0, zf / (zn - zf), zn * zf / (zn - zf)],
                     [0, 0, -1, 0]])
    proj = torch.tensor(clip @ np.linalg.inv(guess), device=dev, dtype=f64)
    flat = target.reshape(-1, 3)
    bad = (flat == 0).all(1)
    pose = torch.tensor(guess, device=dev, dtype=f64)
    pairs, rms = [], []
    for _ in range(c["iterations"]):
        p = eye @ pose.T
        q = p @ proj.T
        a = torch.trunc(q[:, 0] / q[:, 3] * (w * 0.5) + w * 0.5).long() - 10
        b = (h - 1 - torch.trunc(q[:, 1] / q[:, 3] * (h * 0.5) + h * 0.5).long()) - 10
        a, b = a.clamp(min=0), b.clamp(min=0)
        best = torch.full_like(d, 0.01)
        hit = torch.zeros_like(p[:, :3])
        found = torch.zeros_like(d, dtype=torch.bool)
        for i in range(21):
            for j in range(21):
                at = (b + i) * w + (a + j)
                inside = (b + i < 480) & (a + j < 640) & (at < flat.shape[0])
                at = torch.where(inside, at, torch.zeros_like(at))
                t = flat[at]
                l2 = (t - p[:, :3]).square().sum(1)
                better = inside & ~bad[at] & (l2 < best)
                best = torch.where(better, l2, best)
                hit = torch.where(better[:, None], t, hit)
                found |= better
        src, dst = p[found][:, :3], hit[found]
        ms, md = src.mean(0), dst.mean(0)
        S = ((src - ms).T @ (dst - md)).cpu().numpy()
        (xx, xy, xz), (yx, yy, yz), (zx, zy, zz) = S
        n4 = np.array([[xx + yy + zz, yz - zy, zx - xz, xy - yx], [yz - zy, xx - yy - zz, xy + yx, zx + xz],
                       [zx - xz, xy + yx, yy - xx - zz, yz + zy], [xy - yx, zx + xz, yz + zy, zz - xx - yy]])
        qw, qx, qy, qz = np.linalg.eigh(n4)[1][:, 3]
        R = np.array([[1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qw * qz), 2 * (qx * qz + qw * qy)],
                      [2 * (qx * qy + qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qw * qx)],
                      [2 * (qx * qz - qw * qy), 2 * (qy * qz + qw * qx), 1 - 2 * (qx * qx + qy * qy)]])
        T = np.eye(4)
        T[:3, :3], T[:3, 3] = R, md.cpu().numpy() - R @ ms.cpu().numpy()
        pose = torch.tensor(T, device=dev, dtype=f64) @ pose
        pairs.append(int(found.sum()))
        rms.append(math.sqrt(float(best[found].sum()) / max(1, pairs[-1])))
    out = pose.T.cpu().numpy().reshape(16)
    return {"pose": out, "pose64": out, "pairs": None, "rms": np.array(rms)}


# -------------------------------------------------------------------- scan

class _MeshBuffers:
    """The caller's own mesh on the device: room for any mesh of the scene, and the counts of the last."""

    def __init__(self, lib, volume, voxel_mm, indices):
        verts, idx = {8: (2 << 20, 12 << 20), 4: (10 << 20, 48 << 20), 2: (24 << 20, 48 << 20)}[voxel_mm]
        self.lib, self.volume = lib, volume
        self.stream = torch.cuda.ExternalStream(lib.kifi_volume_stream(volume))
        self.verts = torch.zeros((verts, 3), dtype=torch.float32, device="cuda")
        self.indices = torch.zeros(idx, dtype=torch.int32, device="cuda") if indices else None
        torch.cuda.synchronize()

    def take(self):
        """Mesher::Mesh on the volume, into these buffers."""
        nv, ni, pv, pi = C.c_size_t(), C.c_size_t(), C.c_void_p(), C.c_void_p()
        with_indices = self.indices is not None
        check(self.lib.kifi_mesh_device(self.volume, 1 if with_indices else 0, C.byref(nv), C.byref(ni),
                                        C.byref(pv), C.byref(pi)))
        out = {"counts": np.array([nv.value, ni.value], np.int64), "verts": self.verts}
        with torch.cuda.stream(self.stream):  # after the mesh, before the volume's next work
            self.verts[:nv.value].copy_(_view(pv.value, (nv.value, 3), "<f4", torch.float32))
            if with_indices:
                self.indices[:ni.value].copy_(_view(pi.value, (ni.value,), "<i4", torch.int32))
                out["indices"] = self.indices
        return out


def _prepare_scan(c, seed):
    w, h, n = c["width"], c["height"], c["frames"]
    if c["scene"] == "sphere":
        seq = scenes.sphere_scene(n, seed=_seed(seed), width=w, height=h)
        frames = torch.from_numpy(np.stack(seq.frames).view(np.int16)).cuda()
        w2e = np.stack([seq.world_to_eye_f32(i) for i in range(n)])
        f = 292.5 * w / 320.0
        params = kifi.DepthSensorParams((w, h), (f, f), (w / 2.0, h / 2.0), (0.4, 4.0))
    else:
        frames, poses = _room(seed, w, h, [c["stride"] * k for k in range(n)])
        w2e, params = _w2e(poses), _params(w, h)
    cap = _capacity(c, n)
    s = {"kind": "scan", "c": c, "frames": frames, "w2e": w2e, "params": params,
         "volume": kifi.Volume(c["res"], _side(c), _trunc(c), capacity=cap)}
    if c["out"] == "export":  # the caller's own buffers, page-locked
        wide = s["volume"].key_bits == 64
        most = min(cap, {8: 1 << 20, 4: 8 << 20, 2: 24 << 20}[c["voxel_mm"]])
        s["keys"] = torch.zeros(most, dtype=torch.int64 if wide else torch.int32, pin_memory=True)
        s["values"] = torch.zeros((most, 2), dtype=torch.float32, pin_memory=True)
    else:
        s["mesh"] = _MeshBuffers(_lib.load(), s["volume"].handle, c["voxel_mm"], c["out"] == "mesh")
    return s


def _run_scan(s):
    c, vol, lib = s["c"], s["volume"], _lib.load()
    integrator = kifi.Integrator()
    vol.clear()
    for k in range(c["frames"]):
        integrator.IntegrateDevice(vol, s["frames"][k].data_ptr(), True, s["params"], s["w2e"][k])
    if c["out"] != "export":
        return s["mesh"].take()
    n = C.c_size_t()
    call = lib.kifi_volume_export64 if vol.key_bits == 64 else lib.kifi_volume_export
    check(call(vol.handle, C.c_void_p(s["keys"].data_ptr()), C.c_void_p(s["values"].data_ptr()),
               s["keys"].numel(), C.byref(n)))
    return {"count": n.value, "keys": s["keys"], "values": s["values"]}


# -------------------------------------------------------------------- mesh

def _warm(lib, volume, c, seed):
    """Fuses the room as seen from c["warm"] places into a volume."""
    if not c["warm"]:
        return
    frames, poses = _room(seed, c["width"], c["height"], _warm_numbers(c["warm"]))
    cam, w2e = _camera(c["width"], c["height"]), _w2e(poses)
    torch.cuda.synchronize()
    for k in range(c["warm"]):
        check(lib.kifi_integrate_device(volume, C.c_void_p(frames[k].data_ptr()), 1, C.byref(cam), _ptr(w2e[k])))
        if k % 8 == 7:
            check(lib.kifi_volume_sync(volume))
    check(lib.kifi_volume_sync(volume))


def _prepare_mesh(c, seed):
    vol = kifi.Volume(c["res"], _side(c), _trunc(c), capacity=_capacity(c, c["warm"]))
    _warm(_lib.load(), vol.handle, c, seed)
    return {"kind": "mesh", "c": c, "volume": vol,
            "mesh": _MeshBuffers(_lib.load(), vol.handle, c["voxel_mm"], c["indices"])}


def _run_mesh(s):
    return s["mesh"].take()


# --------------------------------------------------------------- pipelines

def _desc(c, mesh_every, closed):
    d = PipelineDesc()
    d.camera = _camera(c["width"], c["height"])
    d.resolution, d.side_length_m, d.truncation_m = c["res"], _side(c), _trunc(c)
    d.icp_iterations, d.mesh_every, d.mesh_with_indices = c["iterations"], mesh_every, 1
    d.initial_capacity = _capacity(c, c["warm"] + c["frames"])
    d.closed_loop = 1 if closed else 0
    return d


def _prepare_pipeline(c, seed, kind, mesh_every, closed):
    lib = _lib.load()
    d, h = _desc(c, mesh_every, closed), C.c_void_p()
    check(lib.kifi_pipeline_create(C.byref(d), C.byref(h)))
    pipe = _Owned(h, lib.kifi_pipeline_destroy)
    _warm(lib, lib.kifi_pipeline_volume(h), c, seed)
    unique = 2 * c["frames"]
    frames, poses = _room(seed, c["width"], c["height"], list(range(100, 100 + unique)))
    s = {"kind": kind, "c": c, "pipe": pipe, "w2e": _w2e(poses), "order": _back_and_forth(unique), "next": 0,
         "frames": _host_u16(frames) if c.get("feed", "host") == "host" else frames}
    s["at"] = [C.c_void_p(f.data_ptr()) for f in s["frames"]]
    s["mesh"] = _MeshBuffers(lib, lib.kifi_pipeline_volume(h), c["voxel_mm"], True)
    return s


def _frames_of(s):
    for _ in range(s["c"]["frames"]):
        j = s["order"][s["next"] % len(s["order"])]
        s["next"] += 1
        yield j


def _prepare_track(c, seed):
    return _prepare_pipeline(c, seed, "track", c["mesh_every"], False)


def _run_track(s):
    lib, h, c = _lib.load(), s["pipe"].h, s["c"]
    poses = np.zeros((c["frames"], 16), np.float32)
    if c["feed"] == "host":
        for k, j in enumerate(_frames_of(s)):
            check(lib.kifi_pipeline_integrate(h, s["at"][j], 1, _ptr(s["w2e"][j]), _ptr(poses[k])))
    else:
        for j in _frames_of(s):
            check(lib.kifi_pipeline_integrate_device(h, s["at"][j], 1, _ptr(s["w2e"][j])))
    last = np.zeros(16, np.float32)
    check(lib.kifi_pipeline_sync(h, _ptr(last)))
    out = {"pose": last}
    if c["feed"] == "host":
        out["poses"] = poses
    if c["mesh_every"]:
        nv, ni = C.c_size_t(), C.c_size_t()
        check(lib.kifi_pipeline_mesh_counts(h, C.byref(nv), C.byref(ni)))
        out["live_mesh_counts"] = np.array([nv.value, ni.value], np.int64)
    out.update(s["mesh"].take())
    return out


def _prepare_closed(c, seed):
    return _prepare_pipeline(c, seed, "closed", 0, True)


def _run_closed(s):
    lib, h, c = _lib.load(), s["pipe"].h, s["c"]
    poses = np.zeros((c["frames"], 16), np.float32)
    for k, j in enumerate(_frames_of(s)):
        check(lib.kifi_pipeline_integrate(h, s["at"][j], 1, _ptr(s["w2e"][j]), _ptr(poses[k])))
    out = {"poses": poses}
    out.update(s["mesh"].take())
    return out


# ----------------------------------------------------------------- batches

_SIZES = [(320, 240), (512, 424), (640, 480), (1024, 848)]
_VOXELS = [(512, 8), (1024, 4), (2048, 2)]


def _scene_specs(c):
    r = np.random.default_rng(c["spec_seed"])
    out = []
    for _ in range(c["scenes"]):
        (w, h), (res, vox) = _SIZES[int(r.integers(4))], _VOXELS[int(r.integers(3))]
        out.append({"width": w, "height": h, "res": res, "voxel_mm": vox, "iterations": c["iterations"],
                    "frames": c["steps"], "warm": 2})
    return out


def _prepare_batch(c, seed):
    lib, specs = _lib.load(), _scene_specs(c)
    descs = (PipelineDesc * len(specs))(*[_desc(q, 0, False) for q in specs])
    h = C.c_void_p()
    check(lib.kifi_batch_create(descs, len(specs), C.byref(h)))
    batch = _Owned(h, lib.kifi_batch_destroy)
    data = []
    for i, q in enumerate(specs):
        _warm(lib, lib.kifi_batch_volume(h, i), q, seed + 17 * i)
        fr, poses = _room(seed + 17 * i, q["width"], q["height"], list(range(100, 100 + c["steps"] + 2)))
        data.append((fr, _w2e(poses)))
    meshes = [_MeshBuffers(lib, lib.kifi_batch_volume(h, i), q["voxel_mm"], True) for i, q in enumerate(specs)]
    return {"kind": "batch", "c": c, "batch": batch, "data": data, "next": 0, "meshes": meshes,
            "order": _back_and_forth(c["steps"] + 2)}


def _run_batch(s):
    lib, h, n = _lib.load(), s["batch"].h, len(s["data"])
    at, w2e = (C.c_void_p * n)(), np.zeros((n, 16), np.float32)
    for _ in range(s["c"]["steps"]):
        j = s["order"][s["next"] % len(s["order"])]
        s["next"] += 1
        for i, (fr, m) in enumerate(s["data"]):
            at[i] = fr[j].data_ptr()
            w2e[i] = m[j]
        check(lib.kifi_batch_step_device(h, at, _ptr(w2e)))
    check(lib.kifi_batch_sync(h))
    poses = np.zeros((n, 16), np.float32)
    for i in range(n):
        check(lib.kifi_batch_pose(h, i, _ptr(poses[i])))
    return {"poses": poses, "meshes": [m.take() for m in s["meshes"]]}


# ---------------------------------------------------------- pose proposer

def _box_down(frames):
    """(n, h, w) millimetre frames -> (n, 60, 80) metres, the mean of each block's valid depths."""
    n, h, w = frames.shape
    d = (frames.to(torch.int32) & 0xFFFF).to(torch.float64) * 0.001
    d = d.reshape(n, 60, h // 60, 80, w // 80).permute(0, 1, 3, 2, 4).reshape(n, 60, 80, -1)
    valid = (d > 0).sum(-1)
    return torch.where(valid > 0, d.sum(-1) / valid.clamp(min=1), torch.zeros_like(d[..., 0]))


def _pair_inputs(seed, batch):
    """batch network inputs [60, 80, 2] from frame pairs one to three apart."""
    n = (batch + 2) // 3
    small = _box_down(_room(seed, 320, 240, list(range(20, 20 + n + 3)))[0])
    x = torch.stack([torch.stack([small[a], small[a + k]], -1) for a in range(n) for k in (1, 2, 3)])[:batch]
    return x.to(torch.float16).contiguous()


def _prepare_predict(c, seed):
    params, mean, std = proposer.load(WEIGHTS)
    net = proposer.PoseProposer(max_batch=c["batch"])
    net.set_params(params)
    s = {"kind": "predict", "c": c, "net": net, "frames": None}
    if c["pairs"] == 1:
        s["frames"] = _room(seed, 640, 480, [20, 21])[0]
        s["x"] = torch.zeros((c["batch"], 60, 80, 2), dtype=torch.float16, device="cuda")
    else:
        s["x"] = _pair_inputs(seed, c["batch"])
    return s


def _run_predict(s):
    if s["frames"] is not None:
        a, b = s["frames"]
        s["net"].make_input(a.data_ptr(), b.data_ptr(), True, 640, 480, s["x"][0].data_ptr())
    return {"twists": s["net"].predict(s["x"])}


def _network(params):
    """Float64 weights of the four convolutions and two linear layers from the parameter vector."""
    at, out = 0, []
    for cin, cout, kp in [(2, 32, 32), (32, 64, 288), (64, 64, 576), (64, 128, 576)]:
        wt = params[at:at + cout * kp].reshape(cout, kp)
        at += cout * kp
        out += [wt, params[at:at + cout]]
        at += cout
    for rows, cols in [(64, 128), (16, 64)]:
        out += [params[at:at + rows * cols].reshape(rows, cols), params[at + rows * cols:at + rows * cols + rows]]
        at += rows * cols + rows
    return out


def _forward64(net, x):
    a = x.to(torch.float64).permute(0, 3, 1, 2)
    for k, cin in enumerate([2, 32, 64, 64]):
        wt = net[2 * k][:, :9 * cin].reshape(-1, 3, 3, cin).permute(0, 3, 1, 2)
        a = torch.relu(torch.nn.functional.conv2d(a, wt, net[2 * k + 1], stride=2, padding=1))
    a = a.mean((2, 3))
    a = torch.relu(a @ net[8].T + net[9])
    return (a @ net[10].T + net[11])[:, :6]


def _exact_predict(c, seed):
    s = _prepare_predict(c, seed)
    x = s["x"].to(torch.float64)
    if s["frames"] is not None:
        x[0] = torch.stack(list(_box_down(s["frames"])), -1)
    net = _network(torch.tensor(proposer.load(WEIGHTS)[0], device="cuda", dtype=torch.float64))
    return {"twists": _forward64(net, x)}


def _prepare_gradients(c, seed):
    g = torch.Generator().manual_seed(_seed(seed))
    net = proposer.PoseProposer(max_batch=c["batch"])
    params = proposer.init_params(_seed(seed))
    net.set_params(params)
    return {"kind": "gradients", "c": c, "net": net, "params": params, "x": _pair_inputs(seed, c["batch"]),
            "y": torch.randn((c["batch"], 6), generator=g).cuda()}


def _run_gradients(s):
    loss, grads = s["net"].gradients(s["x"], s["y"])
    return {"loss": loss, "gradients": grads}


def _exact_gradients(c, seed):
    s = _prepare_gradients(c, seed)
    p = torch.tensor(s["params"], device="cuda", dtype=torch.float64, requires_grad=True)
    loss = (_forward64(_network(p), s["x"]) - s["y"].to(torch.float64)).square().mean()
    loss.backward()
    return {"loss": float(loss), "gradients": p.grad}


# ------------------------------------------------------------ work and exact

def _seen(w, h, vox):
    """Voxels one room frame touches, about: what its surfaces' voxels come to
    once pixels finer than a voxel share one."""
    px = w * h
    pitch = 2000.0 / (F_PER_W * w)  # millimetres between pixels at 2 m
    return 1.25 * px * 8.0 / (1.0 + 2.5 * (vox / pitch) ** 1.5)


def _fuse_bytes(w, h, vox, new):
    """One frame: its depth, the seen voxels' keys and values read and values
    written, the new ones' keys written."""
    return 2.0 * w * h + 20.0 * _seen(w, h, vox) + 4.0 * new


def _icp_flops(w, h, iterations):
    """Per source and iteration: its transform and projection, the nearest of
    at least 3 x 3 candidates, and Horn's sums."""
    return 170.0 * iterations * ((w + 3) // 4) * h


def work(case):
    c, k = case, case["kind"]
    if k == "icp":
        px = c["width"] * c["height"]
        return {"bytes": px * (16.0 if c["form"] == "points" else 4.0),
                "flops": _icp_flops(c["width"], c["height"], c["iterations"])}
    if k in ("predict", "gradients"):
        macs = 30 * 40 * 18 * 32 + 15 * 20 * 288 * 64 + 8 * 10 * 576 * 64 + 4 * 5 * 576 * 128 + 128 * 64 + 64 * 6
        first = 30 * 40 * 18 * 32
        n = c["batch"]
        data = n * 60 * 80 * 4.0 + 4.0 * 135000
        if k == "predict":
            return {"bytes": data + (2 * 640 * 480 * 2.0 if c["pairs"] == 1 else 0.0), "flops": 2.0 * n * macs}
        return {"bytes": data + 4.0 * 135000, "flops": 2.0 * n * (3 * macs - first)}
    if k == "batch":
        b = f = 0.0
        for q in _scene_specs(c):
            w, h = q["width"], q["height"]
            seen = _seen(w, h, q["voxel_mm"])
            b += c["steps"] * _fuse_bytes(w, h, q["voxel_mm"], 0.1 * seen) + 2 * 12.0 * 1.2 * seen
            f += _icp_flops(w, h, c["iterations"]) * c["steps"]
        return {"bytes": b, "flops": f}
    w, h, vox = c["width"], c["height"], c["voxel_mm"]
    seen = _seen(w, h, vox)
    # the voxels in the volume: what its views see, less what they share
    n = seen * (1.0 + 0.6 * c["warm"] if "warm" in c else 1.0 + 0.05 * c["frames"] * c["stride"])
    mesh = 12.0 * n + 0.3 * n * 12 + (1.5 * n * 4 if c.get("indices", c.get("out") != "verts") else 0.0)
    if k == "mesh":
        return {"bytes": mesh, "flops": 10.0 * n}
    b = c["frames"] * _fuse_bytes(w, h, vox, 0.05 * seen) + (24.0 * n if c.get("out") == "export" else mesh)
    return {"bytes": b, "flops": 60.0 * seen * c["frames"] + (_icp_flops(w, h, c["iterations"]) * c["frames"]
                                                              if "iterations" in c else 0.0)}


def exact(case, seed):
    """ICP poses and residuals, the network's outputs and gradients.  Volumes
    and meshes have none: which voxels exist and which triangles join them
    follow from roundings of the float path."""
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None
