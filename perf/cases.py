"""The work a user has this framework do, one case for each part of it.

    fuse        frames through the per-frame pipeline (tracking, integration, raycast)
    preprocess  one depth frame to filtered pyramid, vertex and normal maps
    associate   the sums of one ICP iteration (Estimate_Combined)
    integrate   one frame into a TSDF volume (Integrate_Tsdf_Data)
    raycast     the model maps of one view (Raycast, Resize_*_Map)
    export      the whole model as points (Extract_Tsdf_Volume)
    odometry    one frame of the RGB-D tracker (Estimate_Isometry_By_RGBD)
    refine      the learned depth refiner, forward
    train       one training step of it

Sizes are those of the synthetic configurations (3deye_gb300/synth.py: 320x240
with 128^3, 640x480 with 512^3), of the tests (160x120 with 64^3) and what lies
between; a seed chooses the scene, the trajectory and the sensor noise.
"""
import ctypes as C
import dataclasses
import importlib
import math
from pathlib import Path

import numpy as np
import torch

tde = importlib.import_module("3deye_gb300")
syn = importlib.import_module("3deye_gb300.synth")
pl = importlib.import_module("3deye_gb300.pipeline")
rg = importlib.import_module("3deye_gb300.rgbd")
rf = importlib.import_module("3deye_gb300.refiner")

I16, F16, F32 = tde.TSDF_I16, tde.TSDF_F16, tde.TSDF_F32
WEIGHTS = Path(tde.__file__).resolve().parent / "weights" / "refiner_640x480.f32"
# (channels of the upsampled or only input, channels of the skip, output channels, how the input is read)
_NET = [(16, 0, 16, ""), (16, 0, 32, "pool"), (32, 0, 32, ""), (32, 0, 48, "pool"), (48, 0, 48, ""),
        (48, 0, 64, "pool"), (64, 0, 64, ""), (64, 48, 48, "up"), (48, 32, 32, "up"), (32, 16, 16, "up")]


def listed():
    return [
        # the smallest reconstruction the tests run, one frame at a time with its pose awaited: latency alone
        {"name": "fuse 160x120 64^3 f32, one", "kind": "fuse", "cols": 160, "rows": 120, "voxels": 64, "fmt": F32,
         "frames": 1, "colour": False, "learned": False, "host": False},
        # the headline: a sensor's frames in pinned host memory, tracked and fused back to back
        {"name": "fuse 640x480 512^3 f16", "kind": "fuse", "cols": 640, "rows": 480, "voxels": 512, "fmt": F16,
         "frames": 16, "colour": False, "learned": False, "host": True},
        # the same with an RGB camera and a colour volume
        {"name": "fuse 640x480 512^3 f16 rgb", "kind": "fuse", "cols": 640, "rows": 480, "voxels": 512, "fmt": F16,
         "frames": 8, "colour": True, "learned": False, "host": True},
        # the same with the learned refiner in place of the bilateral filter
        {"name": "fuse 640x480 512^3 f16 net", "kind": "fuse", "cols": 640, "rows": 480, "voxels": 512, "fmt": F16,
         "frames": 8, "colour": False, "learned": True, "host": True},
        # the stages on their own, as a caller with a loop of its own uses them: filter, pyramid and maps
        {"name": "preprocess 640x480", "kind": "preprocess", "cols": 640, "rows": 480},
        # ... the sums of one ICP iteration
        {"name": "associate 640x480", "kind": "associate", "cols": 640, "rows": 480},
        # ... integration, in the reference's own record, an odd frame and a volume that has been shifted
        {"name": "integrate 611x457 384^3 i16", "kind": "integrate", "cols": 611, "rows": 457, "voxels": 384,
         "fmt": I16, "shifted": True},
        # ... the model's maps
        {"name": "raycast 640x480 512^3 f16", "kind": "raycast", "cols": 640, "rows": 480, "voxels": 512, "fmt": F16,
         "shifted": False},
        # the finished model, once a reconstruction ends (and on every shift, a part of it)
        {"name": "export 512^3 f16", "kind": "export", "nx": 512, "ny": 512, "nz": 512, "fmt": F16, "shifted": False},
        # the second tracker, a frame at a time
        {"name": "odometry 640x480", "kind": "odometry", "cols": 640, "rows": 480, "levels": 4, "graphs": True},
        # the refiner on its own: one frame, and the training batch of its recipe
        {"name": "refine 640x480 b1", "kind": "refine", "cols": 640, "rows": 480, "batch": 1},
        {"name": "train 640x480 b16", "kind": "train", "cols": 640, "rows": 480, "batch": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fuse", "fuse", "fuse", "preprocess", "associate", "integrate", "raycast", "export",
                       "odometry", "refine", "train"])
    cols, rows = _log(rng, 128, 640), _log(rng, 96, 480)
    fmt = rng.choice([I16, F16, F32])
    if kind == "fuse":
        learned = rng.random() < 0.25
        if learned:  # the network pools three times
            cols, rows = cols // 8 * 8, rows // 8 * 8
        return {"kind": kind, "cols": cols, "rows": rows, "voxels": _log(rng, 16, 128) * 4, "fmt": fmt,
                "frames": rng.randint(1, 12), "colour": rng.random() < 0.25, "learned": learned,
                "host": rng.random() < 0.5}
    if kind in ("preprocess", "associate"):
        return {"kind": kind, "cols": cols, "rows": rows}
    if kind in ("integrate", "raycast"):
        return {"kind": kind, "cols": cols, "rows": rows, "voxels": _log(rng, 64, 512), "fmt": fmt,
                "shifted": rng.random() < 0.5}
    if kind == "export":  # depths are the reference's table of chunks
        n = rng.choice([128, 256, 512])
        return {"kind": kind, "nx": _log(rng, 100, 512), "ny": _log(rng, 100, 512), "nz": n, "fmt": fmt,
                "shifted": rng.random() < 0.5}
    if kind == "odometry":
        return {"kind": kind, "cols": cols, "rows": rows, "levels": rng.randint(2, 4), "graphs": rng.random() < 0.7}
    return {"kind": kind, "cols": cols // 8 * 8, "rows": rows // 8 * 8,
            "batch": _log(rng, 1, 8) if kind == "refine" else _log(rng, 2, 16)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _config(case):
    base = syn.CONFIGS["c2"]
    cols, rows, vox = case["cols"], case["rows"], case.get("voxels", 512)
    f = 525.0 * cols / 640.0
    return dataclasses.replace(base, cols=cols, rows=rows, fx=f, fy=f, cx=(cols - 1) / 2.0, cy=(rows - 1) / 2.0,
                               voxels=vox, tsdf_format=case.get("fmt", F16), trunc_m=max(0.03, 3 * 3.0 / vox))


def _intr(cfg):
    return tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)


def _sequence(cfg, seed, n):
    """The seeded scene and trajectory: (scene on the host and device, poses [n, 12])."""
    scene = syn.make_scene(cfg, 1000 + seed % 100003)
    return scene, torch.from_numpy(scene).cuda(), syn.make_trajectory(cfg, 2000 + seed % 100003, n)


def _depth(cfg, scene_d, pose, seed, frame, clean=False):
    """One frame of the synthetic sensor: noisy mm (int16 storage), or noise-free metres."""
    fn = tde.lib.tde_synth_depth
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.POINTER(tde.Intrinsics), C.c_uint32, C.c_uint32, C.c_float,
                   C.c_float, C.c_void_p, C.c_void_p, C.c_void_p]
    mm = torch.empty((cfg.rows, cfg.cols), dtype=torch.int16, device="cuda")
    m = torch.empty((cfg.rows, cfg.cols), dtype=torch.float32, device="cuda")
    p = np.ascontiguousarray(pose, np.float64)
    tde.check(fn(scene_d.data_ptr(), scene_d.shape[0], p.ctypes.data_as(C.c_void_p), C.byref(_intr(cfg)),
                 3000 + seed % 100003, frame, cfg.max_depth_mm / 1000.0, 0.02, mm.data_ptr(), m.data_ptr(),
                 torch.cuda.current_stream().cuda_stream))
    return m if clean else mm


def _rgb(cfg, scene_d, pose):
    out = torch.empty((cfg.rows, cfg.cols, 3), dtype=torch.uint8, device="cuda")
    rg.synth_rgb(scene_d, scene_d.shape[0], pose, _intr(cfg), out, torch.cuda.current_stream())
    return out


def _maps(cfg, depth_m):
    """Vertex and normal maps of a metric depth frame by differences, NaN where a pixel or a neighbour is empty."""
    u = torch.arange(cfg.cols, device="cuda", dtype=torch.float32)[None, :]
    v = torch.arange(cfg.rows, device="cuda", dtype=torch.float32)[:, None]
    z = torch.where(depth_m > 0, depth_m, torch.nan)
    vm = torch.stack([z * (u - cfg.cx) / cfg.fx, z * (v - cfg.cy) / cfg.fy, z], -1)
    n = torch.full_like(vm, torch.nan)
    dx, dy = vm[1:-1, 2:] - vm[1:-1, :-2], vm[2:, 1:-1] - vm[:-2, 1:-1]
    c = torch.cross(dy, dx, dim=-1)
    n[1:-1, 1:-1] = c / c.norm(dim=-1, keepdim=True)
    return vm.contiguous(), torch.where(torch.isnan(vm), torch.nan, n).contiguous()


def _sdf(scene, x, y, z):
    d = torch.full(torch.broadcast_shapes(x.shape, y.shape, z.shape), 1e9, device="cuda")
    for p in scene.tolist():
        a = p[1:]
        if p[0] == 0:  # the ground: what lies above it is free
            s = -(a[0] * x + a[1] * y + a[2] * z + a[3])
        elif p[0] == 1:
            s = ((x - a[0]) ** 2 + (y - a[1]) ** 2 + (z - a[2]) ** 2).sqrt() - a[3]
        else:
            q = [(w - 0.5 * (a[k] + a[k + 3])).abs() - 0.5 * (a[k + 3] - a[k]) for k, w in enumerate((x, y, z))]
            out = (q[0].clamp(min=0) ** 2 + q[1].clamp(min=0) ** 2 + q[2].clamp(min=0) ** 2).sqrt()
            s = out + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0)
        d = torch.minimum(d, s)
    return d


def _volume(scene, pose, cfg, dims, fmt, origin, seed):
    """What a volume holds some dozen frames into a reconstruction: free space at 1 and a noisy band about the
    surface inside the view, nothing (value 0, weight 0) elsewhere.  Returns (values float [z, y, x], weights int32,
    the packed volume)."""
    nx, ny, nz = dims
    size = cfg.volume_m
    g = torch.Generator(device="cuda").manual_seed(seed)
    R = torch.tensor(pose[:9].reshape(3, 3), dtype=torch.float32, device="cuda")
    t = [float(v) for v in pose[9:]]
    x = ((torch.arange(nx, device="cuda") + 0.5) * (size / nx))[None, None, :]
    y = ((torch.arange(ny, device="cuda") + 0.5) * (size / ny))[None, :, None]
    f, w = [], []
    for z0 in range(0, nz, 32):
        z = ((torch.arange(z0, min(z0 + 32, nz), device="cuda") + 0.5) * (size / nz))[:, None, None]
        s = _sdf(scene, x, y, z)
        c = [R[0, k] * (x - t[0]) + R[1, k] * (y - t[1]) + R[2, k] * (z - t[2]) for k in range(3)]
        seen = (c[2] > 0.1) & ((cfg.fx * c[0] / c[2]).abs() < 0.5 * cfg.cols) & \
            ((cfg.fy * c[1] / c[2]).abs() < 0.5 * cfg.rows) & (s > -cfg.trunc_m)
        v = s / cfg.trunc_m
        v = torch.where(v > 1, 1.0, v + 0.03 * torch.randn(v.shape, device="cuda", generator=g)).clamp(-1, 1)
        f.append(torch.where(seen, v, 0.0))
        w.append(torch.where(seen, torch.randint(1, 60, v.shape, device="cuda", generator=g, dtype=torch.int32), 0))
    f, w = torch.cat(f), torch.cat(w).to(torch.int32)
    if fmt == I16:
        q = (f * 32767.0).to(torch.int32)
        f, rec = q.float() / 32767.0, ((q & 0xFFFF) | (w << 16))
    elif fmt == F16:
        h = f.half()
        f, rec = h.float(), ((h.view(torch.int16).to(torch.int32) & 0xFFFF) | (w << 16))
    else:
        rec = f
    roll = (origin[2], origin[1], origin[0])
    rec = torch.roll(rec, roll, (0, 1, 2)).contiguous().view(-1)
    vol = rec.view(torch.uint8)
    if fmt == F32:
        vol = torch.cat([vol, torch.roll(w, roll, (0, 1, 2)).to(torch.int16).contiguous().view(-1).view(torch.uint8)])
    return f, w, vol


def _records(vol, fmt, n):
    """A packed volume as the values it holds: whole records, or the float plane and the weights."""
    return [vol[:4 * n].view(torch.float32), vol[4 * n:].view(torch.int16)] if fmt == F32 else [vol.view(torch.int32)]


def _origin(case, dims):
    return (dims[0] // 3, dims[1] // 5 + 1, dims[2] // 2) if case["shifted"] else (0, 0, 0)


class _Raw:
    """Device memory of a pipeline, for torch.as_tensor: the tensor keeps this object, and so the pipeline, alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_Raw(owner, ptr, shape, typestr), device="cuda")


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _prepare_fuse(case, seed):
    cfg = _config(case)
    k = max(case["frames"] + 1, 8)
    _, scene_d, traj = _sequence(cfg, seed, k)
    depth = torch.stack([_depth(cfg, scene_d, traj[i], seed, i) for i in range(k)])
    rgb = torch.stack([_rgb(cfg, scene_d, traj[i]) for i in range(k)]) if case["colour"] else None
    torch.cuda.synchronize()
    p = pl.Pipeline(cfg, traj[0])
    net = None
    if case["learned"]:
        net = rf.Refiner(1, cfg.rows, cfg.cols)
        net.set_params(np.fromfile(WEIGHTS, np.float32))
        p.set_refiner(net)
    if case["colour"]:
        p.enable_color()
    if case["host"]:
        depth = depth.cpu().pin_memory()
        rgb = rgb.cpu().pin_memory() if rgb is not None else None
    n = case["frames"]
    vp, _ = p.volume()
    vox = case["voxels"] ** 3
    if case["fmt"] == F32:
        vol = [_view(p, vp, (vox,), "<f4"), _view(p, vp + 4 * vox, (vox,), "<i2")]
    else:
        vol = [_view(p, vp, (vox,), "<i4")]
    if case["colour"]:
        vol.append(_view(p, p.color_volume(), (vox,), "<i4"))
    vm, nm = p.model_maps(0)
    shape = (cfg.rows, cfg.cols, 3)
    s = {"case": case, "cfg": cfg, "p": p, "net": net, "depth": depth, "rgb": rgb,
         # there and back along the trajectory, so that each frame is one step from the last
         "order": [*range(k), *range(k - 2, 0, -1)], "at": 0,
         "pose": torch.zeros((n, 12), dtype=torch.float64).pin_memory(),
         "status": torch.zeros(n, dtype=torch.int32).pin_memory(),
         "maps": [_view(p, vm, shape, "<f4"), _view(p, nm, shape, "<f4")], "volume": vol}
    for _ in range(k):  # the model that the next frames are tracked against
        _enqueue(s, 0)
    p.sync()
    return s


def _enqueue(s, slot):
    i = s["order"][s["at"] % len(s["order"])]
    s["at"] += 1
    on_device = not s["case"]["host"]
    pose, status = s["pose"].data_ptr() + 96 * slot, s["status"].data_ptr() + 4 * slot
    if s["rgb"] is not None:
        s["p"].enqueue_rgbd(s["depth"][i].data_ptr(), s["rgb"][i].data_ptr(), on_device, pose, status)
    else:
        s["p"].enqueue(s["depth"][i].data_ptr(), on_device, pose, status)


def _run_fuse(s):
    for slot in range(s["case"]["frames"]):
        _enqueue(s, slot)
    s["p"].sync()  # the poses are in host memory
    return {"pose": s["pose"], "status": s["status"], "maps": s["maps"], "volume": s["volume"]}


def _prepare_preprocess(case, seed):
    cfg = _config(case)
    _, scene_d, traj = _sequence(cfg, seed, 2)
    i0 = _intr(cfg)
    lv = [i0.level(l) for l in range(3)]
    depth = [torch.empty((i.rows, i.cols), dtype=torch.int16, device="cuda") for i in lv]
    v = [torch.empty((i.rows, i.cols, 3), dtype=torch.float32, device="cuda") for i in lv]
    n = [torch.empty_like(x) for x in v]
    ptrs = (C.c_void_p * 3)(*[d.data_ptr() for d in depth])
    return {"case": case, "cfg": cfg, "raw": _depth(cfg, scene_d, traj[0], seed, 0), "lv": lv, "depth": depth, "v": v,
            "n": n, "ptrs": ptrs}


def _run_preprocess(s):
    lib, cfg, stream = tde.lib, s["cfg"], torch.cuda.current_stream().cuda_stream
    tde.check(lib.tde_bilateral_pyramid(s["raw"].data_ptr(), s["ptrs"], 3, cfg.cols, cfg.rows, cfg.sigma_space,
                                        cfg.sigma_color, cfg.max_depth_mm, stream))
    for i, d, v, n in zip(s["lv"], s["depth"], s["v"], s["n"]):
        tde.check(lib.tde_vertex_map(d.data_ptr(), v.data_ptr(), C.byref(i), stream))
        tde.check(lib.tde_normal_map(v.data_ptr(), n.data_ptr(), i.cols, i.rows, stream))
    return {"depth": s["depth"], "v": s["v"], "n": s["n"]}


def _inputs_associate(case, seed):
    """Current maps (noisy) at one pose, model maps (clean, global frame) at the one before; the current pose starts
    from the model's."""
    cfg = _config(case)
    _, scene_d, traj = _sequence(cfg, seed, 2)
    vm, nm = _maps(cfg, _depth(cfg, scene_d, traj[0], seed, 0, clean=True))
    vc, nc = _maps(cfg, _depth(cfg, scene_d, traj[1], seed, 1, clean=True))
    g = torch.Generator(device="cuda").manual_seed(seed)
    vc = vc * (1 + 0.001 * torch.randn(vc.shape[:2], device="cuda", generator=g))[..., None]
    R = torch.tensor(traj[0][:9].reshape(3, 3), dtype=torch.float32, device="cuda")
    t = torch.tensor(traj[0][9:], dtype=torch.float32, device="cuda")
    return cfg, traj, vc.contiguous(), nc, (vm @ R.T + t).contiguous(), (nm @ R.T).contiguous()


def _prepare_associate(case, seed):
    cfg, traj, vc, nc, vm, nm = _inputs_associate(case, seed)
    R, t = traj[0][:9].reshape(3, 3), traj[0][9:]
    g = torch.empty(tde.lib.tde_estimate_combined_gbuf_floats(cfg.cols, cfg.rows), device="cuda")
    return {"case": case, "cfg": cfg, "maps": (vc, nc, vm, nm), "R": tde.mat3(R), "t": tde.vec3(t),
            "Ri": tde.mat3(R.T.copy()), "g": g, "m": torch.empty(27, device="cuda"), "intr": _intr(cfg)}


def _run_associate(s):
    cfg = s["cfg"]
    tde.check(tde.lib.tde_estimate_combined(*[m.data_ptr() for m in s["maps"]], C.byref(s["R"]), C.byref(s["t"]),
                                            C.byref(s["Ri"]), C.byref(s["t"]), C.byref(s["intr"]), cfg.dist_thresh,
                                            cfg.angle_thresh, s["g"].data_ptr(), s["m"].data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
    return s["m"]


def _prepare_integrate(case, seed):
    cfg = _config(case)
    dims = (case["voxels"],) * 3
    scene, scene_d, traj = _sequence(cfg, seed, 2)
    origin = _origin(case, dims)
    _, _, vol = _volume(scene, traj[0], cfg, dims, case["fmt"], origin, seed)
    return {"case": case, "cfg": cfg, "vol": vol, "rb": tde.round_buffer(dims, (cfg.volume_m,) * 3, origin),
            "depth": _depth(cfg, scene_d, traj[1], seed, 1), "intr": _intr(cfg), "cell": tde.vec3([cfg.cell] * 3),
            "scaled": torch.empty((cfg.rows, cfg.cols), device="cuda"),
            "Ri": tde.mat3(traj[1][:9].reshape(3, 3).T.copy()), "t": tde.vec3(traj[1][9:])}


def _run_integrate(s):
    lib, cfg, stream = tde.lib, s["cfg"], torch.cuda.current_stream().cuda_stream
    tde.check(lib.tde_scale_depth(s["depth"].data_ptr(), s["scaled"].data_ptr(), C.byref(s["intr"]), stream))
    tde.check(lib.tde_integrate_tsdf(s["scaled"].data_ptr(), s["vol"].data_ptr(), s["case"]["fmt"], cfg.trunc_m,
                                     C.byref(s["Ri"]), C.byref(s["t"]), C.byref(s["intr"]), C.byref(s["cell"]),
                                     C.byref(s["rb"]), cfg.max_weight, stream))
    return {"scaled": s["scaled"], "volume": _records(s["vol"], s["case"]["fmt"], s["case"]["voxels"] ** 3)}


def _prepare_raycast(case, seed):
    cfg = _config(case)
    dims = (case["voxels"],) * 3
    scene, _, traj = _sequence(cfg, seed, 2)
    origin = _origin(case, dims)
    _, _, vol = _volume(scene, traj[0], cfg, dims, case["fmt"], origin, seed)
    size = [(cfg.rows >> l, cfg.cols >> l, 3) for l in range(3)]
    return {"case": case, "cfg": cfg, "vol": vol, "rb": tde.round_buffer(dims, (cfg.volume_m,) * 3, origin),
            "intr": _intr(cfg), "cell": tde.vec3([cfg.cell] * 3), "R": tde.mat3(traj[1][:9]), "t": tde.vec3(traj[1][9:]),
            "v": [torch.empty(x, device="cuda") for x in size], "n": [torch.empty(x, device="cuda") for x in size]}


def _run_raycast(s):
    lib, cfg, stream = tde.lib, s["cfg"], torch.cuda.current_stream().cuda_stream
    v, n = s["v"], s["n"]
    tde.check(lib.tde_raycast(s["vol"].data_ptr(), s["case"]["fmt"], v[0].data_ptr(), n[0].data_ptr(), C.byref(s["t"]),
                              C.byref(s["R"]), cfg.trunc_m, C.byref(s["intr"]), C.byref(s["rb"]), C.byref(s["cell"]),
                              stream))
    for l in (1, 2):
        c, r = cfg.cols >> (l - 1), cfg.rows >> (l - 1)
        tde.check(lib.tde_resize_vertex_map(v[l - 1].data_ptr(), v[l].data_ptr(), c, r, stream))
        tde.check(lib.tde_resize_normal_map(n[l - 1].data_ptr(), n[l].data_ptr(), c, r, stream))
    return {"v": v, "n": n}


def _inputs_export(case, seed):
    cfg = _config({"cols": 640, "rows": 480, "voxels": max(case["nx"], case["ny"], case["nz"])})
    dims = (case["nx"], case["ny"], case["nz"])
    scene, _, traj = _sequence(cfg, seed, 1)
    return (cfg, dims, *_volume(scene, traj[0], cfg, dims, case["fmt"], _origin(case, dims), seed))


def _prepare_export(case, seed):
    cfg, dims, _, _, vol = _inputs_export(case, seed)
    rb = tde.round_buffer(dims, (cfg.volume_m,) * 3, _origin(case, dims))
    n = _capacity(dims)
    return {"case": case, "vol": vol, "cell": tde.Point3f(*[cfg.volume_m / d for d in dims]), "rb": rb,
            "scratch": torch.empty(tde.lib.tde_extract_tsdf_volume_scratch_bytes(C.byref(rb)), dtype=torch.uint8,
                                   device="cuda"),
            "points": torch.zeros((n, 4), device="cuda"), "weights": torch.zeros(n, device="cuda"),
            "count": torch.zeros(1, dtype=torch.int32, device="cuda")}


def _capacity(dims):
    """Room for the points of a model, as a caller that extracts one after another keeps it."""
    return dims[0] * dims[1] * dims[2] // 64


def _run_export(s):
    tde.check(tde.lib.tde_extract_tsdf_volume(s["vol"].data_ptr(), s["case"]["fmt"], C.byref(s["rb"]), s["cell"],
                                              s["scratch"].data_ptr(), s["scratch"].numel(), s["points"].data_ptr(),
                                              s["weights"].data_ptr(), s["weights"].numel(), s["count"].data_ptr(),
                                              torch.cuda.current_stream().cuda_stream))
    n = int(s["count"].item())  # how many of the points are the model's
    return {"points": s["points"], "weights": s["weights"], "count": n}


def _inputs_odometry(case, seed):
    cfg = dataclasses.replace(_config(case), voxels=512)
    k = 6
    _, scene_d, traj = _sequence(cfg, seed, k)
    return cfg, [_depth(cfg, scene_d, traj[i], seed, i) for i in range(k)], [_rgb(cfg, scene_d, traj[i])
                                                                             for i in range(k)]


def _prepare_odometry(case, seed):
    cfg, depth, rgb = _inputs_odometry(case, seed)
    torch.cuda.synchronize()
    tr = rg.RgbdTracker(_intr(cfg), rg.default_params(case["levels"]), graphs=case["graphs"])
    k = len(depth)
    s = {"case": case, "tr": tr, "depth": depth, "rgb": rgb, "order": [*range(k), *range(k - 2, 0, -1)], "at": 0}
    _run_odometry(s)
    _run_odometry(s)
    tr.stream.synchronize()
    return s


def _run_odometry(s):
    i = s["order"][s["at"] % len(s["order"])]
    s["at"] += 1
    here = torch.cuda.current_stream()
    s["tr"].stream.wait_stream(here)  # the frames come from the caller's stream
    s["tr"].track(s["depth"][i], s["rgb"][i])
    here.wait_stream(s["tr"].stream)  # and the pose is used there
    return {"pose": s["tr"].pose, "status": s["tr"].status}


def _inputs_net(case, seed):
    """Frames of the sensor, their targets (the noise-free depth, as a fused model gives it) and weights: the committed
    ones for inference, for training those of a run a few steps old (the first layers as they are drawn, a small
    head)."""
    cfg = _config(case)
    _, scene_d, traj = _sequence(cfg, seed, case["batch"])
    raw = torch.stack([_depth(cfg, scene_d, traj[i], seed, i) for i in range(case["batch"])])
    clean = torch.stack([_depth(cfg, scene_d, traj[i], seed, i, clean=True) for i in range(case["batch"])])
    tgt = torch.where(clean <= 4.0, (clean * 1000).round(), 0.0).to(torch.int16)
    if case["kind"] == "refine":
        return cfg, raw, tgt, np.fromfile(WEIGHTS, np.float32)
    r = np.random.RandomState(seed % 100003)
    th = [math.sqrt(2 / 27) * r.standard_normal(16 * 27), np.zeros(16)]
    for ca, cb, co, _ in _NET:
        th += [math.sqrt(2 / (9 * (ca + cb))) * r.standard_normal(co * 9 * (ca + cb)), np.zeros(co)]
    th += [0.05 * r.standard_normal(16), np.zeros(1)]
    return cfg, raw, tgt, np.concatenate(th).astype(np.float32)


def _prepare_net(case, seed):
    cfg, raw, tgt, th = _inputs_net(case, seed)
    net = rf.Refiner(case["batch"], cfg.rows, cfg.cols)
    net.set_params(th)
    return {"case": case, "net": net, "raw": raw, "tgt": tgt, "out": torch.empty(raw.shape, device="cuda")}


def _run_refine(s):
    s["net"].forward_ptr(s["raw"].data_ptr(), s["case"]["batch"], 0, s["out"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _run_train(s):
    s["net"].train_step_ptr(s["raw"].data_ptr(), s["tgt"].data_ptr(), s["case"]["batch"], 1e-4,
                            torch.cuda.current_stream().cuda_stream)
    return s["net"].grads()


_PREPARE = {"fuse": _prepare_fuse, "preprocess": _prepare_preprocess, "associate": _prepare_associate,
            "integrate": _prepare_integrate, "raycast": _prepare_raycast, "export": _prepare_export,
            "odometry": _prepare_odometry, "refine": _prepare_net, "train": _prepare_net}
_RUN = {"fuse": _run_fuse, "preprocess": _run_preprocess, "associate": _run_associate, "integrate": _run_integrate,
        "raycast": _run_raycast, "export": _run_export, "odometry": _run_odometry, "refine": _run_refine,
        "train": _run_train}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "export":  # every record once; 20 bytes for each of about one voxel in 250
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (6 if case["fmt"] == F32 else 4) + n // 250 * 20, "flops": 0}
    px = case["cols"] * case["rows"]
    pyramid = px * (1 + 1 / 4 + 1 / 16)
    filt = px * 169 * 8 + pyramid * 49 * 20      # bilateral window, normal window
    pair = 150                                   # association and 28 products of a pixel
    if kind == "preprocess":
        return {"bytes": 2 * px + pyramid * (2 + 24), "flops": filt}
    if kind == "associate":
        return {"bytes": 48 * px + 108, "flops": pair * px}
    if kind in ("fuse", "integrate", "raycast"):
        rec = 6 if case["fmt"] == F32 else 4
        seen = 0.03 * case["voxels"] ** 3        # records a frame changes (measured over 600 frames at 512^3)
        ray = 2.5 * px * rec                     # distinct records that the rays meet (the same)
        if kind == "integrate":
            return {"bytes": 6 * px + 2 * seen * rec, "flops": 30 * seen}
        if kind == "raycast":
            return {"bytes": ray + 24 * pyramid, "flops": 30 * 20 * px}
        icp = pair * (10 * px + 5 * px / 4 + 4 * px / 16)
        one = {"bytes": 2 * px + 2 * seen * rec + ray + 24 * pyramid, "flops": filt + icp + 30 * seen + 600 * px}
        if case["colour"]:
            one["bytes"] += 3 * px + 0.002 * case["voxels"] ** 3 * 8
        if case["learned"]:
            one["flops"] += rf.conv_flops(case["rows"], case["cols"]) - px * 169 * 8
        return {k: v * case["frames"] for k, v in one.items()}
    if kind == "odometry":
        steps = [7, 7, 7, 10]
        f = sum(n * 2 * px / 4 ** l for l, n in enumerate(steps[:case["levels"]]))
        return {"bytes": 5 * px + 2 * 4 * px + 96, "flops": f * 80}
    b = case["batch"]
    flops = rf.conv_flops(case["rows"], case["cols"], b, train=kind == "train")
    return {"bytes": (6 if kind == "refine" else 4) * px * b + 4 * rf.param_count() * (1 if kind == "refine" else 4),
            "flops": flops + (1 if kind == "refine" else 2) * 2 * 27 * 16 * px * b}


# ---------------------------------------------------------------------------
# exact: the same in 64 bits, with torch alone
# ---------------------------------------------------------------------------
def _exact_preprocess(case, seed):
    cfg = _config(case)
    _, scene_d, traj = _sequence(cfg, seed, 2)
    d = (_depth(cfg, scene_d, traj[0], seed, 0).to(torch.int32) & 0xFFFF).double()
    H, W = d.shape
    pad = torch.nn.functional.pad
    inside = torch.zeros_like(d)
    inside[:H - 1, :W - 1] = 1  # the window ends before the last row and column
    dp, ip = pad(d, (6,) * 4), pad(inside, (6,) * 4)
    s1, s2 = torch.zeros_like(d), torch.zeros_like(d)
    for dy in range(13):
        for dx in range(13):
            t, m = dp[dy:dy + H, dx:dx + W], ip[dy:dy + H, dx:dx + W]
            w = m * torch.exp(-(((dx - 6) ** 2 + (dy - 6) ** 2) * 0.5 / cfg.sigma_space ** 2 +
                                (d - t) ** 2 * 0.5 / cfg.sigma_color ** 2))
            s1 += t * w
            s2 += w
    f = (s1 / s2).round()
    f = torch.where(f > cfg.max_depth_mm, 0.0, f)
    depth, v, n = [], [], []
    i0 = _intr(cfg)
    for l in range(3):
        it = i0.level(l)
        if l:
            src, h, w_ = f, it.rows, it.cols
            sp = pad(src, (2, 3, 2, 3))
            ctr = src[0:2 * h:2, 0:2 * w_:2]
            tot, cnt = torch.zeros_like(ctr), torch.zeros_like(ctr)
            for dy in range(5):
                for dx in range(5):
                    t = sp[dy:dy + 2 * h:2, dx:dx + 2 * w_:2]
                    ok = (t != 0) & ((t - ctr).abs() < int(3 * cfg.sigma_color))
                    tot += torch.where(ok, t, 0.0)
                    cnt += ok
            f = torch.where(ctr != 0, torch.floor((tot + torch.floor(cnt / 2)) / cnt.clamp(min=1)), 0.0)
        z = torch.where(f != 0, f / 1000, torch.nan)
        u = torch.arange(it.cols, device="cuda", dtype=torch.float64)[None, :]
        y = torch.arange(it.rows, device="cuda", dtype=torch.float64)[:, None]
        vm = torch.stack([z * (u - it.cx) / it.fx, z * (y - it.cy) / it.fy, z], -1)
        depth.append(f.to(torch.int16))
        v.append(vm)
        n.append(_exact_normals(vm))
    return {"depth": depth, "v": v, "n": n}


def _exact_normals(vm):
    H, W, _ = vm.shape
    p = torch.nn.functional.pad(vm.permute(2, 0, 1), (3,) * 4, value=float("nan"))
    s1, s2, cnt = torch.zeros_like(vm), torch.zeros((H, W, 3, 3), dtype=torch.float64, device="cuda"), 0
    for dy in range(7):
        for dx in range(7):
            o = p[:, dy:dy + H, dx:dx + W].permute(1, 2, 0) - vm
            ok = ~torch.isnan(o[..., :1])
            o = torch.where(ok, o, 0.0)
            s1 += o
            s2 += o[..., :, None] * o[..., None, :]
            cnt = cnt + ok[..., 0]
    good = ~torch.isnan(vm[..., 0]) & (cnt >= 24)
    c = s2 - s1[..., :, None] * s1[..., None, :] / cnt.clamp(min=1)[..., None, None]
    c = c / c.abs().amax((-1, -2), keepdim=True).clamp(min=1e-300)
    # the smallest eigenvalue in closed form, its vector from the rows' cross products
    q = c.diagonal(dim1=-2, dim2=-1).sum(-1) / 3
    e = torch.eye(3, dtype=torch.float64, device="cuda")
    b = c - q[..., None, None] * e
    pp = (b.square().sum((-1, -2)) / 6).sqrt().clamp(min=1e-300)
    r = (torch.linalg.det(b / pp[..., None, None]) / 2).clamp(-1, 1)
    m = c - (q + 2 * pp * torch.cos(torch.acos(r) / 3 + 2 * math.pi / 3))[..., None, None] * e
    x = torch.stack([torch.cross(m[..., i, :], m[..., j, :], dim=-1) for i, j in ((0, 1), (0, 2), (1, 2))], -2)
    k = x.square().sum(-1).argmax(-1)
    nv = torch.gather(x, -2, k[..., None, None].expand(H, W, 1, 3))[..., 0, :]
    nv = nv / nv.norm(dim=-1, keepdim=True)
    nv = torch.where((nv * vm).sum(-1, keepdim=True) > 0, -nv, nv)
    return torch.where(good[..., None], nv, torch.nan)


def _exact_associate(case, seed):
    cfg, traj, vc, nc, vm, nm = _inputs_associate(case, seed)
    vc, nc, vm, nm = (x.double().reshape(-1, 3) for x in (vc, nc, vm, nm))
    R = torch.tensor(traj[0][:9].reshape(3, 3), dtype=torch.float32, device="cuda").double()
    t = torch.tensor(traj[0][9:], dtype=torch.float32, device="cuda").double()
    keep = ~torch.isnan(nc[:, 0])
    vg, ng = vc[keep] @ R.T + t, nc[keep] @ R.T
    c = (vg - t) @ R  # the model's camera
    u, v = (cfg.fx * c[:, 0] / c[:, 2] + cfg.cx).round(), (cfg.fy * c[:, 1] / c[:, 2] + cfg.cy).round()
    ok = (c[:, 2] > 0) & (u >= 0) & (v >= 0) & (u < cfg.cols) & (v < cfg.rows)
    vg, ng = vg[ok], ng[ok]
    j = (v[ok] * cfg.cols + u[ok]).long()
    vp, np_ = vm[j], nm[j]
    d = vp - vg
    ok = ~torch.isnan(np_[:, 0]) & (d.square().sum(1) <= cfg.dist_thresh ** 2) & \
        (torch.cross(ng, np_, dim=1).square().sum(1) < cfg.angle_thresh ** 2)
    vg, np_, d = vg[ok], np_[ok], d[ok]
    row = torch.cat([torch.cross(vg, np_, dim=1), np_, (np_ * d).sum(1, keepdim=True)], 1)
    A = row.T @ row
    return torch.stack([A[i, k] for i in range(6) for k in range(i, 7)])


def _exact_integrate(case, seed):
    """The scaled depth, and the values where the volume holds floats (whole records have no such value)."""
    cfg = _config(case)
    dims = (case["voxels"],) * 3
    scene, scene_d, traj = _sequence(cfg, seed, 2)
    raw = _depth(cfg, scene_d, traj[1], seed, 1).double()
    u = torch.arange(cfg.cols, device="cuda", dtype=torch.float64)[None, :]
    y = torch.arange(cfg.rows, device="cuda", dtype=torch.float64)[:, None]
    scaled = raw / 1000 * (((u - cfg.cx) / cfg.fx) ** 2 + ((y - cfg.cy) / cfg.fy) ** 2 + 1).sqrt()
    if case["fmt"] != F32:
        return {"scaled": scaled, "volume": [None]}
    origin = _origin(case, dims)
    f, w, _ = _volume(scene, traj[0], cfg, dims, F32, origin, seed)
    f, w = f.double(), w.double()
    n = case["voxels"]
    g = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * cfg.cell
    t = traj[1][9:]
    X, Y = (g - t[0])[None, None, :], (g - t[1])[None, :, None]
    R = traj[1][:9].reshape(3, 3)
    for z0 in range(0, n, 32):
        Z = (g[z0:z0 + 32] - t[2])[:, None, None]
        c = [R[0, k] * X + R[1, k] * Y + R[2, k] * Z for k in range(3)]
        pu, pv = (cfg.fx * c[0] / c[2] + cfg.cx).round(), (cfg.fy * c[1] / c[2] + cfg.cy).round()
        ok = (c[2] > 0) & (pu >= 0) & (pu < cfg.cols) & (pv >= 0) & (pv < cfg.rows)
        D = scaled.reshape(-1)[torch.where(ok, pv * cfg.cols + pu, 0).long()]
        s = D - (X * X + Y * Y + Z * Z).sqrt()
        ok = ok & (D != 0) & (s >= -cfg.trunc_m)
        F, Wt = f[z0:z0 + 32], w[z0:z0 + 32]
        f[z0:z0 + 32] = torch.where(ok, F + ((s / cfg.trunc_m).clamp(max=1) - F) / (Wt + 1), F)
        w[z0:z0 + 32] = torch.where(ok, (Wt + 1).clamp(max=cfg.max_weight), Wt)
    roll = (origin[2], origin[1], origin[0])
    return {"scaled": scaled, "volume": [torch.roll(f, roll, (0, 1, 2)).reshape(-1),
                                         torch.roll(w, roll, (0, 1, 2)).to(torch.int16).reshape(-1)]}


def _exact_export(case, seed):
    cfg, dims, f, w, _ = _inputs_export(case, seed)
    step = {512: 256, 256: 128, 128: 64}[dims[2]] // 2
    cell = torch.tensor([cfg.volume_m / d for d in dims], dtype=torch.float32, device="cuda").double()
    live = (w != 0) & (f != 1)
    s = torch.where(live, torch.sign(f), 0.0)
    pts, wts = [], []
    for z0 in range(0, dims[2], step):
        b = s[z0:z0 + step]
        for q, dim in enumerate((2, 1, 0)):  # +x, +y, +z; [z, y, x]
            k = b.shape[dim] - 1
            at = torch.nonzero(b.narrow(dim, 0, k) * b.narrow(dim, 1, k) < 0)
            at[:, dim] += 1
            at[:, 0] += z0
            # in the order of the voxel that the crossing leaves
            pts.append((at.flip(1).double() + 0.5) * cell)
            wts.append(w[at[:, 0], at[:, 1], at[:, 2]])
    pts, wts, cap = torch.cat(pts), torch.cat(wts), _capacity(dims)
    n = min(cap, pts.shape[0])
    points = torch.zeros((cap, 4), dtype=torch.float64, device="cuda")
    points[:n, :3], points[:n, 3] = pts[:n], 1
    weights = torch.zeros(cap, dtype=torch.float64, device="cuda")
    weights[:n] = wts[:n]
    return {"points": points, "weights": weights, "count": int(pts.shape[0])}


def _exact_odometry(case, seed):
    cfg, depth, rgb = _inputs_odometry(case, seed)
    i0, L = _intr(cfg), case["levels"]

    def pyramid(k):
        c = rgb[k].to(torch.int64)
        I, D = [(c[..., 0] * 4899 + c[..., 1] * 9617 + c[..., 2] * 1868 + 8192) >> 14], [depth[k].double() * 0.001]
        for l in range(1, L):
            h, w = cfg.rows >> l, cfg.cols >> l
            p = I[-1][:2 * h, :2 * w].reshape(h, 2, w, 2)
            I.append((p.sum((1, 3)) + 2) >> 2)
            D.append(D[-1][0:2 * h:2, 0:2 * w:2])
        return I, D

    (Ip, Dp), (Ic, Dc) = pyramid(1), pyramid(2)
    T = torch.eye(4, dtype=torch.float64)
    for l in reversed(range(L)):
        it = i0.level(l)
        h, w = it.rows, it.cols
        a = Ic[l].double()
        gx, gy = torch.zeros_like(a), torch.zeros_like(a)
        r0, r1, r2 = a[:-2], a[1:-1], a[2:]
        gx[1:-1, 1:-1] = (r0[:, 2:] + 2 * r1[:, 2:] + r2[:, 2:]) - (r0[:, :-2] + 2 * r1[:, :-2] + r2[:, :-2])
        gy[1:-1, 1:-1] = (r2[:, :-2] + 2 * r2[:, 1:-1] + r2[:, 2:]) - (r0[:, :-2] + 2 * r0[:, 1:-1] + r0[:, 2:])
        u = torch.arange(w, device="cuda", dtype=torch.float64)[None, :].expand(h, w).reshape(-1)
        v = torch.arange(h, device="cuda", dtype=torch.float64)[:, None].expand(h, w).reshape(-1)
        z = Dp[l].reshape(-1)
        sel = (z > 0) & (z < 35)
        u, v, z, ip = u[sel], v[sel], z[sel], Ip[l].reshape(-1)[sel].double()
        X = torch.stack([z * (u - it.cx) / it.fx, z * (v - it.cy) / it.fy, z], 1)
        for _ in range((7, 7, 7, 10)[l]):
            R, t = T[:3, :3].cuda(), T[:3, 3].cuda()
            P = X @ R.T + t
            pu = (it.fx * P[:, 0] / P[:, 2] + it.cx).round()
            pv = (it.fy * P[:, 1] / P[:, 2] + it.cy).round()
            ok = (P[:, 2] > 0) & (pu >= 0) & (pv >= 0) & (pu < w) & (pv < h)
            j = torch.where(ok, pv * w + pu, 0).long()
            z2, dx, dy = Dc[l].reshape(-1)[j], gx.reshape(-1)[j], gy.reshape(-1)[j]
            ok = ok & (z2 > 0) & (z2 < 35) & ((P[:, 2] - z2).abs() < 0.07) & (dx * dx + dy * dy >= 6400)
            if int(ok.sum()) < 6:
                continue
            P, dx, dy, r = P[ok], dx[ok], dy[ok], (Ic[l].reshape(-1)[j].double() - ip)[ok]
            wt = 1 / (r.square().mean().sqrt() + r.abs())
            v0, v1 = wt * 0.125 * it.fx / P[:, 2] * dx, wt * 0.125 * it.fy / P[:, 2] * dy
            g = torch.stack([v0, v1, -(v0 * P[:, 0] + v1 * P[:, 1]) / P[:, 2]], 1)
            J = torch.cat([torch.cross(P, g, dim=1), g], 1)
            x = torch.linalg.solve((J.T @ J).cpu(), -(J.T @ (wt * r)).cpu())
            K = torch.zeros((3, 3), dtype=torch.float64)
            K[0, 1], K[0, 2], K[1, 0], K[1, 2], K[2, 0], K[2, 1] = -x[2], x[1], x[2], -x[0], -x[1], x[0]
            E = torch.linalg.matrix_exp(K)
            T[:3, 3] = E @ T[:3, 3] + x[3:]
            T[:3, :3] = E @ T[:3, :3]
    return {"pose": torch.cat([T[:3, :3].reshape(-1), T[:3, 3]]), "status": None}


def _net64(theta, raw):
    """The network in 64 bits: (refined metres, valid)."""
    F = torch.nn.functional
    at = 0

    def take(*shape):
        nonlocal at
        n = int(np.prod(shape))
        at += n
        return theta[at - n:at].reshape(shape)

    d = (raw.to(torch.int32) & 0xFFFF).double()[:, None] * 0.001
    n, _, h, w = d.shape
    nb = F.unfold(d, 3, padding=1).reshape(n, 9, h, w)
    valid = nb > 0
    feat = torch.stack([torch.where(valid & (d > 0), (nb - d) * 100, 0.0), valid.double(), nb], 2).reshape(n, 27, h, w)
    w1, b1 = take(16, 27), take(16)
    x = torch.relu(torch.einsum("ok,nkhw->nohw", w1, feat) + b1[:, None, None])
    skip = []
    for ca, cb, co, how in _NET:
        wt, b = take(co, 3, 3, ca + cb), take(co)
        if how == "pool":
            skip.append(x)
            x = F.max_pool2d(x, 2)
        elif how == "up":
            x = torch.cat([x.repeat_interleave(2, 2).repeat_interleave(2, 3), skip.pop()], 1)
        x = torch.relu(F.conv2d(x, wt.permute(0, 3, 1, 2), b, padding=1))
    hw, hb = take(16), take(1)
    r = torch.einsum("o,nohw->nhw", hw, x) + hb
    d = d[:, 0]
    return torch.where(d > 0, d + 0.01 * r, 0.0), d > 0


def _exact_refine(case, seed):
    _, raw, _, th = _inputs_net(case, seed)
    theta = torch.from_numpy(th).double().cuda()
    with torch.no_grad():
        return torch.cat([_net64(theta, raw[i:i + 1])[0] for i in range(case["batch"])])


def _exact_train(case, seed):
    _, raw, tgt, th = _inputs_net(case, seed)
    theta = torch.from_numpy(th).double().cuda().requires_grad_()
    for i in range(case["batch"]):  # the loss is a sum over the batch: its gradients add up
        out, valid = _net64(theta, raw[i:i + 1])
        t = (tgt[i:i + 1].to(torch.int32) & 0xFFFF).double() * 0.001
        (torch.where(valid & (t > 0), (out - t).abs(), 0.0).sum() / raw.numel()).backward()
    return theta.grad


def exact(case, seed):
    # Tracked frames ("fuse") would take minutes in 64 bits.  A raycast's hits are decided by the sign of the samples
    # that its 32-bit march meets; in 64 bits other rays hit or miss at the outlines, so there is no value to compare.
    fn = {"preprocess": _exact_preprocess, "associate": _exact_associate, "integrate": _exact_integrate,
          "export": _exact_export, "odometry": _exact_odometry, "refine": _exact_refine,
          "train": _exact_train}.get(case["kind"])
    return fn(case, seed) if fn else None
