"""Benchmark of the per-frame KinectFusion pipeline (plain path).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload: the 640x480 / 512^3 FP16+u16 TSDF sequence (seeded synthetic scene,
orbit and Kinect noise; frames = W + K of one contiguous sequence; one step
is one frame).  The first W frames warm up (frame 0 initialises the model).

Reported (one JSON line, rank 0):
  value      frames/s with the depth frames already resident in HBM;
  e2e        frames/s through the C-ABI pipeline with depth in pinned host
             memory: every step copies its frame host->device and the frame's
             pose device->host inside the timed region;
  roofline   the dominant kernel, the ICP iteration: 48 B per pixel of
             algorithmic traffic over its time per iteration, against
             MEASURED_PEAKS.json hbm_gbs; `kernels` adds the integration
             sweep (4 B/voxel read + 4 B/voxel written for the voxels the
             update touches, counted live) and the raycast;
  cpu_baseline  the CPU oracle of the same pipeline on this host's cores;
  learned_refine, color_volume, model_export, cyclic_volume, config1
             the refiner in place of the bilateral filter, RGB-D frames with
             the colour volume, the whole-model export and shading, the
             640x480 / 512^3 corridor with the volume following the camera,
             and the 100-frame 320x240 / 128^3 FP32 sequence (GPU and CPU);
  ate_m      against the ground truth and, over the first --f64-frames
             frames, against the full-FP64 oracle pipeline run on the host.
N > 1 runs independent replicas (sequence seed = rank): scaling "weak".

--impl reference runs the CPU implementation of the path (the oracle port:
the reference's OpenCL kernels cannot run on this host -- no CPU OpenCL
runtime -- and its host library does not build) on rank 0.
"""
from __future__ import annotations

import argparse
import ctypes as C
import importlib
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "frames/s 640x480 @512³ TSDF (plain vs learned-refine, equal ATE); kernel GB/s vs HBM"
WORKLOAD = "c2"
WORKLOAD_DESC = "640x480 depth, 512^3 TSDF over 3 m (fp16+u16), ICP 3 levels 10/5/4"
DATA = "synthetic (seeded procedural scene, orbit, Kinect noise; sequence seed 0 + rank)"


def bench_config(ws: int, nframes: int) -> dict:
    """The `config` object both arms print (the same workload, frames and seed)."""
    return {"workload": WORKLOAD_DESC, "global_batch": 1, "frames": nframes, "sequence_seed": 0,
            "l2": "inputs larger than L2 (512 MiB TSDF volume swept every frame)",
            "parallelism": "replicas" if ws > 1 else "single"}


def load_synth():
    """synth.py (the seeded scene, trajectory and seed rules) loaded by file
    path, so that the CPU arm never imports the package (which maps the CUDA
    library)."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("tde_synth_standalone", ROOT / "3deye_gb300" / "synth.py")
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod  # dataclasses resolve their module by name
    spec.loader.exec_module(mod)
    return mod


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=590)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--cpu-frames", type=int, default=40,
                    help="frames of the CPU baseline sample (about 11 s on 16 cores; capped by the sequence length)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--skip", default="", help="comma list of further passes to leave out (color, learned, cyclic, "
                                               "config1, rgbd), e.g. for a short profiling run")
    ap.add_argument("--f64-frames", type=int, default=30,
                    help="leading frames of the sequence the full-FP64 oracle also runs (ATE of the GPU trajectory "
                         "against it)")
    ap.add_argument("--refiner-weights", default=str(ROOT / "3deye_gb300" / "weights" / "refiner_640x480.f32"),
                    help="trained refiner for the learned-refine line (skipped when the file is absent)")
    return ap.parse_args()


def dist_init(args):
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch
        import torch.distributed as dist
        gpu = torch.cuda.is_available()
        if gpu:
            torch.cuda.set_device(local)
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        # replicas exchange only the barrier and the max of their times: NCCL
        # between the GPU arm's ranks, gloo for the CPU reference arm (and on
        # hosts without a GPU)
        dist.init_process_group("nccl" if args.impl == "ours" and gpu else "gloo")
    return ws, rank, local


class ClockSampler:
    """SM clocks and clock-event (throttle) reasons of the benchmark's GPU,
    read through NVML (libnvidia-ml, by ctypes) in a polling thread every
    ~0.5 ms, so that even a timed region of a few milliseconds holds samples;
    nvidia-smi at 50 ms where NVML cannot be loaded.  `window()` brackets a
    timed region: summary(window=True) covers only the samples inside it."""

    REASONS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown", 0x40: "hw_thermal_slowdown",
               0x80: "hw_power_brake_slowdown"}

    def __init__(self, torch_device):
        self.dev = torch_device
        self.samples = []  # (perf_counter, sm_mhz, reasons mask)
        self.max_mhz = None
        self.windows = []
        self._stop = threading.Event()
        self._nvml = None
        self._h = None
        self.source = None

    def _open_nvml(self):
        import torch
        nv = C.CDLL("libnvidia-ml.so.1")
        if nv.nvmlInit_v2() != 0:
            raise OSError("nvmlInit failed")
        h = C.c_void_p()
        uuid = getattr(torch.cuda.get_device_properties(self.dev), "uuid", None)
        ok = False
        if uuid is not None:
            ok = nv.nvmlDeviceGetHandleByUUID(f"GPU-{uuid}".encode(), C.byref(h)) == 0
        if not ok and nv.nvmlDeviceGetHandleByIndex_v2(self.dev.index or 0, C.byref(h)) != 0:
            raise OSError("no NVML handle")
        self.reason_fn = getattr(nv, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            nv.nvmlDeviceGetCurrentClocksThrottleReasons
        mx = C.c_uint()
        if nv.nvmlDeviceGetMaxClockInfo(h, 1, C.byref(mx)) == 0:  # NVML_CLOCK_SM
            self.max_mhz = float(mx.value)
        self._nvml, self._h = nv, h

    def _poll_nvml(self):
        nv, h = self._nvml, self._h
        mhz, mask = C.c_uint(), C.c_ulonglong()
        while not self._stop.is_set():
            if nv.nvmlDeviceGetClockInfo(h, 1, C.byref(mhz)) == 0 and self.reason_fn(h, C.byref(mask)) == 0:
                self.samples.append((time.perf_counter(), float(mhz.value), int(mask.value)))
            time.sleep(0.0005)

    def _poll_smi(self):
        q = "clocks.sm,clocks.max.sm,clocks_event_reasons.active"
        proc = subprocess.Popen(["nvidia-smi", "-i", str(self.dev.index or 0), f"--query-gpu={q}",
                                 "--format=csv,noheader,nounits", "-lms", "50"], stdout=subprocess.PIPE,
                                stderr=subprocess.DEVNULL, text=True)
        self._proc = proc
        for line in proc.stdout:
            f = [x.strip() for x in line.split(",")]
            try:
                self.samples.append((time.perf_counter(), float(f[0]), int(f[2], 16)))
                self.max_mhz = float(f[1])
            except (ValueError, IndexError):
                continue

    def __enter__(self):
        try:
            self._open_nvml()
            self.source = "nvml"
            target = self._poll_nvml
        except (OSError, AttributeError):
            self.source = "nvidia-smi"
            target = self._poll_smi
        self._thread = threading.Thread(target=target, daemon=True)
        self._thread.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        if getattr(self, "_proc", None):
            self._proc.terminate()
        self._thread.join(timeout=5)

    def window(self):
        sampler = self

        class _W:
            def __enter__(self):
                self.t0 = time.perf_counter()
                return self

            def __exit__(self, *exc):
                sampler.windows.append((self.t0, time.perf_counter()))
        return _W()

    def summary(self, window=True):
        pts = list(self.samples)
        if window and self.windows:
            pts = [p for p in pts if any(a <= p[0] <= b for a, b in self.windows)]
        if not pts:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": [], "samples": 0, "source": self.source}
        reasons = sorted({name for _, _, m in pts for bit, name in self.REASONS.items() if m & bit})
        return {"sm_mhz": statistics.median(p[1] for p in pts), "sm_max_mhz": self.max_mhz, "reasons": reasons,
                "samples": len(pts), "source": self.source}


def load_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def load_peaks_bf16():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"burst": float(d["bf16_tflops"]), "sustained": float(d["bf16_tflops_sustained"]), "kind": "measured"}
    return {"burst": 1900.0, "sustained": 1700.0, "kind": "fallback"}


def load_traffic(name="integrate_c2_traffic.json"):
    """DRAM bytes of one ncu capture of a kernel, from the committed summary."""
    p = ROOT / "profiles" / name
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            return None
    return None


# ---------------------------------------------------------------------------
def make_frames(tde, syn, cfg, nframes, seed_k, dev, corridor=False):
    """Render the sequence on the GPU sensor; returns (device uint16 [n,H,W], gt poses)."""
    import numpy as np
    import torch
    s_scene, s_traj, s_noise = syn.seeds(seed_k)
    if corridor:
        scene = syn.make_corridor_scene(cfg, s_scene)
        traj = syn.make_corridor_trajectory(cfg, s_traj, nframes)
    else:
        scene = syn.make_scene(cfg, s_scene)
        traj = syn.make_trajectory(cfg, s_traj, nframes)
    tde.lib.tde_synth_depth.restype = C.c_int
    tde.lib.tde_synth_depth.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.POINTER(tde.Intrinsics), C.c_uint32,
                                        C.c_uint32, C.c_float, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p]
    d_scene = torch.from_numpy(scene).to(dev)
    intr = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    frames = torch.empty((nframes, cfg.rows, cfg.cols), dtype=torch.uint16, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    for i in range(nframes):
        pose = np.ascontiguousarray(traj[i])
        tde.check(tde.lib.tde_synth_depth(d_scene.data_ptr(), scene.shape[0], pose.ctypes.data_as(C.c_void_p),
                                          C.byref(intr), s_noise, i, cfg.max_depth_mm / 1000.0, 0.02,
                                          frames[i].data_ptr(), None, stream))
    torch.cuda.synchronize()
    return frames, traj, scene


def barrier_sync(ws):
    import torch
    gpu = torch.cuda.is_available()
    if gpu:
        torch.cuda.synchronize()
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()
        if gpu:
            torch.cuda.synchronize()


def max_over_ranks(ws, x):
    """The largest of the ranks' values (every rank gets it)."""
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device="cuda" if dist.get_backend() == "nccl" else "cpu")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def cpu_baseline_run(cfg, frames_np, traj, nframes, threads=None):
    """Oracle pipeline on the host's cores (or `threads` of them) over the
    first frames; frame 0 (model initialisation) is untimed."""
    from oracle import oracle as orc
    from oracle.pipeline import OraclePipeline
    cores = orc.set_threads(threads or os.cpu_count() or 1)
    op = OraclePipeline(cfg, traj[0])
    op.process(frames_np[0])
    t0 = time.perf_counter()
    for i in range(1, nframes + 1):
        op.process(frames_np[i])
    dt = time.perf_counter() - t0
    orc.set_threads(os.cpu_count() or 1)
    return nframes / dt, cores, dt


def fp64_oracle_poses(cfg, frames_np, traj):
    """Poses of the full-FP64 oracle pipeline (FP64 TSDF, integration,
    raycast, ICP terms and solve) on the given frames, all host cores."""
    from oracle import oracle as orc
    from oracle.pipeline import OraclePipelineF64
    orc.set_threads(os.cpu_count() or 1)
    op = OraclePipelineF64(cfg, traj[0])
    poses = [op.process(f) for f in frames_np]
    return __import__("numpy").array(poses), int(sum(op.lost))


def cpu_legs(cfg, frames, traj, n_all, n_one, n_f64, label):
    """The CPU side of one workload, on rank 0: the oracle pipeline timed on
    every host core and on one core, and the FP64 oracle's poses of the first
    n_f64 frames (for the GPU trajectory's ATE against it)."""
    fnp = frames[: max(n_all, n_one, n_f64 - 1) + 1].cpu().numpy()
    v, cores, dt = cpu_baseline_run(cfg, fnp, traj, n_all)
    v1, _, dt1 = cpu_baseline_run(cfg, fnp, traj, n_one, threads=1)
    t0 = time.perf_counter()
    f64, f64_lost = fp64_oracle_poses(cfg, fnp[:n_f64], traj)
    cpu = {"value": round(v, 4), "unit": "frames/s", "cores": cores, "kind": "port",
           "sample": f"frames 1-{n_all} of the same sequence through the CPU oracle pipeline ({label}, {cores} "
                     f"OpenMP threads, {dt:.1f} s)",
           "one_core": {"value": round(v1, 4), "unit": "frames/s", "cores": 1,
                        "sample": f"frames 1-{n_one}, 1 thread, {dt1:.1f} s"}}
    return cpu, {"poses": f64, "lost": f64_lost, "frames": n_f64, "s": time.perf_counter() - t0}


def ate_vs_fp64(pl, est, f64):
    if not f64:
        return {}
    m = f64["frames"]
    return {"vs_fp64_oracle": round(pl.ate_rmse(est[:m], f64["poses"]), 9),
            "vs_fp64_oracle_frames": f"0-{m - 1} (the full-FP64 oracle pipeline on the same frames, "
                                     f"{f64['s']:.1f} s on the host; tracking lost there on {f64['lost']} frames)"}


def model_export(tde, torch, cp, cfg, dev, reps=5):
    """Whole-model export of the fused sequence (Extract_Tsdf_Volume on the
    512^3 volume, Extract_Color_Volume of its points, Generate_Image of the
    model), each timed with CUDA events on the launching stream after a
    warm-up call; and the host-side export through the pipeline API."""
    import numpy as np
    vptr, rb = cp.volume()
    s = torch.cuda.current_stream(dev)
    sp = C.c_void_p(s.cuda_stream)
    lib = tde.lib
    scratch = torch.empty(lib.tde_extract_tsdf_volume_scratch_bytes(C.byref(rb)), dtype=torch.uint8, device=dev)
    cnt = torch.zeros(1, dtype=torch.int32, device=dev)
    c = float(np.float32(cfg.volume_m) / np.float32(cfg.voxels))
    cell = tde.Point3f(c, c, c)
    tde.check(lib.tde_extract_tsdf_volume(C.c_void_p(vptr), cfg.tsdf_format, C.byref(rb), cell, tde.ptr(scratch),
                                          scratch.numel(), None, None, 0, tde.ptr(cnt), sp))
    npts = int(cnt.item())
    pts = torch.empty((max(npts, 1), 4), dtype=torch.float32, device=dev)
    wts = torch.empty(max(npts, 1), dtype=torch.float32, device=dev)
    cols = torch.empty((max(npts, 1), 4), dtype=torch.uint8, device=dev)
    img = torch.empty((cfg.rows, cfg.cols, 3), dtype=torch.uint8, device=dev)

    def timed(fn):
        fn()
        torch.cuda.synchronize(dev)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        for _ in range(reps):
            fn()
        e1.record(s)
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1) / reps

    ext_ms = timed(lambda: tde.check(lib.tde_extract_tsdf_volume(
        C.c_void_p(vptr), cfg.tsdf_format, C.byref(rb), cell, tde.ptr(scratch), scratch.numel(), tde.ptr(pts),
        tde.ptr(wts), npts, tde.ptr(cnt), sp)))
    col_ms = timed(lambda: tde.check(lib.tde_extract_color_volume(
        C.c_void_p(cp.color_volume()), C.byref(rb), tde.ptr(pts), npts, cell, tde.ptr(cols), sp)))
    light = tde.LightSource(tde.Point3f(*(float(v) for v in cp.pose()[9:])), 1)
    vm, nm = cp.model_maps(0)
    ren_ms = timed(lambda: tde.check(lib.tde_generate_image(C.c_void_p(vm), C.c_void_p(nm), cfg.cols, cfg.rows,
                                                            C.byref(light), tde.ptr(img), sp)))
    t0 = time.perf_counter()
    _, _, _, n_host = cp.extract_volume(capacity=npts)
    host_ms = (time.perf_counter() - t0) * 1e3
    rec = tde.lib.tde_tsdf_volume_bytes(cfg.tsdf_format, C.byref(rb))
    # the extraction must read every voxel record once and write 20 B per
    # point (point + weight); the count pass reads the volume and keeps 16
    # predicate bits per 4 voxels, which the scatter reads instead
    alg = rec + npts * 20
    hbm, peak_kind = load_peaks()
    return {"points": npts, "host_points": n_host,
            "extract_tsdf_volume": {"ms": round(ext_ms, 4), "alg_bytes": int(alg),
                                    "achieved_gbs": round(alg / (ext_ms * 1e-3) / 1e9, 1), "peak": hbm,
                                    "frac": round(alg / (ext_ms * 1e-3) / 1e9 / hbm, 4),
                                    "launches": 3,
                                    "note": "count (reads the 512^3 fp16+u16 volume, stores 2 B of predicate bits "
                                            "per 4 voxels), scan, scatter (reads the bits, writes the points)"},
            "extract_color_volume_ms": round(col_ms, 4),
            "generate_image_ms": round(ren_ms, 4),
            "host_export_ms": round(host_ms, 2),
            "note": "after the RGB-D sequence; host export = count + scatter + colour lookup + D2H of points, "
                    "weights and colours through tde_pipeline_extract_volume (wall clock)"}


def cyclic_run(tde, syn, pl, torch, dev, rank):
    """The cyclic-volume workload: 600 frames of 640x480 along a 12 m corridor,
    a 512^3 fp16+u16 volume over 3 m re-centred (slab extracted to host memory
    and cleaned, origins advanced) whenever the point 1.5 m ahead of the camera
    leaves the central 0.8 m.  Frames are enqueued back to back; after
    enqueueing frame i the host waits for frame i-1's pose (downloaded by the
    enqueue) and decides on a shift from it, so the decision is one frame late
    and the GPU keeps frame i in flight meanwhile.  Wall clock over the whole
    sequence."""
    import numpy as np
    cfg = syn.CONFIGS["c3"]
    n = cfg.frames
    frames, traj, _ = make_frames(tde, syn, cfg, n, rank, dev, corridor=True)
    p = pl.Pipeline(cfg, traj[0], use_graphs=True)
    stream = torch.cuda.ExternalStream(p.stream)
    poses = torch.zeros((n, 12), dtype=torch.float64).pin_memory()
    done = [torch.cuda.Event() for _ in range(n)]
    cell = cfg.volume_m / cfg.voxels
    offset, off_at = np.zeros(3), np.zeros((n, 3))
    shift_s, points = [], 0
    torch.cuda.synchronize(dev)
    t0 = time.perf_counter()
    for i in range(n):
        p.enqueue(frames[i].data_ptr(), True, poses[i].data_ptr())
        done[i].record(stream)
        off_at[i] = offset
        if i == 0:
            continue
        done[i - 1].synchronize()
        prev = poses[i - 1].numpy().copy()
        prev[9:] -= offset - off_at[i - 1]  # into the current volume frame
        delta = p.shift_needed_for(prev, 0.4)
        if delta.any():
            ts = time.perf_counter()
            _, _, k = p.shift(delta)
            shift_s.append(time.perf_counter() - ts)
            points += k
            offset = offset + delta * cell
    torch.cuda.synchronize(dev)
    total = time.perf_counter() - t0
    p.close()
    del frames
    est = poses.numpy().copy()
    est[:, 9:] += off_at
    return {"value": round(n / total, 2), "unit": "frames/s", "frames": n,
            "shifts": len(shift_s), "points_extracted": int(points),
            "ms_per_shift": round(1e3 * float(np.mean(shift_s)), 3) if shift_s else None,
            "ate_m": round(pl.ate_rmse(est, traj), 6),
            "note": "640x480, 512^3 fp16+u16 over 3 m following a 12 m corridor walk; frames enqueued back to "
                    "back, each shift decided from the previous frame's pose while the next frame runs; a shift "
                    "synchronises, extracts the outgoing slab to host memory, cleans it, advances the origins, "
                    "re-casts the model and updates the frame graphs; wall clock"}


def config1_run(tde, syn, pl, torch, dev, rank, ws, with_cpu):
    """The small configuration (100 frames of 320x240, 128^3 FP32 over 2 m,
    ICP 10/5/4): GPU frames/s over frames 10-99 resident in HBM, the
    trajectory's ATE against the ground truth and against the full-FP64
    oracle over all 100 frames, and the CPU oracle pipeline on every host core
    and on one core."""
    cfg = syn.CONFIGS["c1"]
    n, W = cfg.frames, 10
    frames, traj, _ = make_frames(tde, syn, cfg, n, rank, dev)
    cpu, f64 = (None, None)
    if with_cpu:
        cpu, f64 = cpu_legs(cfg, frames, traj, n - 1, 10, n, "320x240, 128^3 FP32")
    p = pl.Pipeline(cfg, traj[0], use_graphs=True)
    poses = torch.zeros((n, 12), dtype=torch.float64, pin_memory=True)
    stat = torch.zeros(n, dtype=torch.int32, pin_memory=True)
    base, fb = frames.data_ptr(), cfg.rows * cfg.cols * 2
    for i in range(W):
        p.enqueue(base + i * fb, True, poses[i].data_ptr(), stat[i].data_ptr())
    p.sync()
    st = torch.cuda.ExternalStream(p.stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier_sync(ws)
    e0.record(st)
    for i in range(W, n):
        p.enqueue(base + i * fb, True, poses[i].data_ptr(), stat[i].data_ptr())
    e1.record(st)
    p.sync()
    ms = max_over_ranks(ws, e0.elapsed_time(e1))
    p.close()
    est = poses.numpy().copy()
    out = {"workload": "320x240 depth, 128^3 TSDF over 2 m (fp32+u16), ICP 3 levels 10/5/4, 100 frames",
           "value": round(ws * (n - W) / (ms * 1e-3), 2), "unit": "frames/s", "timed_frames": f"{W}-{n - 1}",
           "ms_per_step": round(ms / (n - W), 5),
           "ate_m": {"vs_ground_truth": round(pl.ate_rmse(est, traj), 6),
                     "frames_tracking_lost": int((stat.numpy() != 0).sum()), **ate_vs_fp64(pl, est, f64)},
           "cpu_baseline": cpu}
    del frames
    return out


def color_pass(tde, pl, torch, cfg, traj, frames, W, n, ws, dev, pose_a):
    """Pass D: RGB-D frames with the colour volume on (Integrate_Colors), then
    the whole-model export.  Synthetic colour: a deterministic pattern of the
    pixel and frame index, resident in HBM beside the depth frames."""
    import numpy as np
    K = n - W
    base, fbytes = frames.data_ptr(), cfg.rows * cfg.cols * 2
    cp = pl.Pipeline(cfg, traj[0], use_graphs=True)
    cp.enable_color(max_weight=128)
    i32 = torch.int32
    yy, xx = torch.meshgrid(torch.arange(cfg.rows, device=dev, dtype=i32), torch.arange(cfg.cols, device=dev, dtype=i32),
                            indexing="ij")
    kk = torch.arange(n, device=dev, dtype=i32).view(n, 1, 1)
    rgb_frames = torch.empty((n, cfg.rows, cfg.cols, 3), dtype=torch.uint8, device=dev)
    rgb_frames[..., 0] = (xx + 3 * kk) % 256
    rgb_frames[..., 1] = (yy + 5 * kk) % 256
    rgb_frames[..., 2] = ((xx + yy) % 256).expand(n, -1, -1)
    cbase, cfb = rgb_frames.data_ptr(), cfg.rows * cfg.cols * 3
    for i in range(W):
        cp.enqueue_rgbd(base + i * fbytes, cbase + i * cfb, True)
    cp.sync()
    cstream = torch.cuda.ExternalStream(cp.stream)
    h0, h1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier_sync(ws)
    h0.record(cstream)
    for i in range(W, n):
        cp.enqueue_rgbd(base + i * fbytes, cbase + i * cfb, True)
    h1.record(cstream)
    cp.sync()
    c_ms = max_over_ranks(ws, h0.elapsed_time(h1))
    c_launches = cp.launches_per_frame()
    pose_c = cp.pose()
    export = model_export(tde, torch, cp, cfg, dev)
    cp.close()
    del rgb_frames
    color = {"value": round(ws * K / (c_ms * 1e-3), 2), "unit": "frames/s", "ms_per_step": round(c_ms / K, 5),
             "gpu_launches": c_launches * K, "same_trajectory_as_plain": bool(np.array_equal(pose_c, pose_a)),
             "note": "RGB-D frames (synthetic colour pattern, resident in HBM): the plain pipeline plus the colour "
                     "volume update at the model surface after each raycast (brick-culled, 4 B per voxel)"}
    return color, export


def rgbd_pass(tde, syn, torch, cfg, dev, ws, rank, with_cpu, pairs=48, warm=4):
    """Pass R: dense RGB-D odometry (Estimate_Isometry_By_RGBD) between
    consecutive frames of a rendered sequence with colour: per frame the
    intensity/depth pyramid and Sobel derivatives, then 4 levels of
    Gauss-Newton (7, 7, 7, 10 steps) against the previous frame.  Depth
    (noisy, uint16 mm) and RGB frames are rendered by the GPU sensor and
    resident in HBM."""
    import numpy as np
    rg = importlib.import_module("3deye_gb300.rgbd")
    n = pairs + warm + 1
    frames, traj, scene = make_frames(tde, syn, cfg, n, rank + 17, dev)
    intr = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    d_scene = torch.from_numpy(np.ascontiguousarray(scene, np.float64)).to(dev)
    rgb = torch.empty((n, cfg.rows, cfg.cols, 3), dtype=torch.uint8, device=dev)
    for i in range(n):
        rg.synth_rgb(d_scene, scene.shape[0], traj[i], intr, rgb[i])
    torch.cuda.synchronize()
    poses = torch.zeros((n, 12), dtype=torch.float64, device=dev)
    stats = torch.zeros(n, dtype=torch.int32, device=dev)

    def timed(graphs):
        tr = rg.RgbdTracker(intr, device=dev, graphs=graphs)
        s = tr.stream

        def step(i):
            tr.track(frames[i], rgb[i])
            with torch.cuda.stream(s):
                poses[i].copy_(tr.pose, non_blocking=True)
                stats[i:i + 1].copy_(tr.status, non_blocking=True)
        tr.track(frames[0], rgb[0])
        for i in range(1, warm + 1):
            step(i)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.synchronize()
        barrier_sync(ws)
        e0.record(s)
        for i in range(warm + 1, n):
            step(i)
        e1.record(s)
        s.synchronize()
        return max_over_ranks(ws, e0.elapsed_time(e1)), tr, poses.cpu().numpy()
    ms_eager, _, est_eager = timed(False)
    ms, tr, _ = timed(True)
    od = tr.od
    est = poses.cpu().numpy()
    st = stats.cpu().numpy()
    et, er = [], []
    for i in range(1, n):
        Rp, tp = traj[i - 1][:9].reshape(3, 3), traj[i - 1][9:]
        Rc, tc = traj[i][:9].reshape(3, 3), traj[i][9:]
        gR, gt = Rc.T @ Rp, Rc.T @ (tp - tc)
        Re = est[i][:9].reshape(3, 3) @ gR.T
        et.append(np.linalg.norm(est[i][9:] - gt))
        er.append(np.degrees(np.arccos(np.clip((np.trace(Re) - 1) / 2, -1, 1))))
    levels = 4
    # the pose, one launch for the steps of the levels of up to 16 blocks of 2048 pixels, two for each other step
    large = [l for l in range(levels) if (cfg.cols >> l) * (cfg.rows >> l) > 16 * 2048]
    launches = ((1 + (levels - 1) + levels) + 1 + int(len(large) < levels) +
                2 * sum(int(od.params.iters[l]) for l in large))
    out = {"value": round(ws * pairs / (ms * 1e-3), 2), "unit": "frames/s", "ms_per_step": round(ms / pairs, 5),
           "ms_per_step_without_graphs": round(ms_eager / pairs, 5), "gpu_launches": launches * pairs,
           "graph_poses_equal_eager": bool(np.array_equal(est, est_eager)),
           "relative_pose_error": {"mean_translation_m": round(float(np.mean(et)), 6),
                                   "mean_rotation_deg": round(float(np.mean(er)), 5),
                                   "mean_step_translation_m": round(float(np.mean(
                                       [np.linalg.norm(traj[i][9:] - traj[i - 1][9:]) for i in range(1, n)])), 6),
                                   "frames_without_a_solved_step": int(((st[1:] & 2) == 0).sum())},
           "note": "640x480 noisy depth + rendered texture, resident in HBM; per frame: intensity, 4-level "
                   "pyramid, Sobel derivatives and 31 Gauss-Newton steps (those of the levels of up to 16 blocks in "
                   "one cluster launch, 17 of them here; 2 passes each on the others, the 6x6 solve in the second "
                   "pass's last block), replayed from CUDA graphs (RgbdTracker)"}
    if with_cpu:
        from oracle import oracle as orc
        fr = frames[:4].view(torch.int16).cpu().numpy().view(np.uint16)
        cols = rgb[:4].cpu().numpy()
        lv = [orc.rgbd_levels(fr[i], cols[i], levels) for i in range(4)]
        io = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)

        def cpu_fps(pairs):
            t0 = time.perf_counter()
            for i in range(1, pairs + 1):
                orc.rgbd_odometry(lv[i - 1], lv[i], io, [7, 7, 7, 10], [10.0] * 4)
            return pairs / (time.perf_counter() - t0)
        cores = orc.set_threads(os.cpu_count() or 1)
        fps_all = cpu_fps(3)
        orc.set_threads(1)
        fps_one = cpu_fps(1)
        orc.set_threads(os.cpu_count() or 1)
        out["cpu_baseline"] = {"value": round(fps_all, 3), "unit": "frames/s", "cores": cores, "kind": "port",
                               "sample": "odometry of 3 frame pairs (pyramids prepared beforehand), OpenMP over "
                                         "pixel rows",
                               "one_core": {"value": round(fps_one, 3), "unit": "frames/s", "cores": 1,
                                            "sample": "1 frame pair"}}
    return out


def run_ours(args, ws, rank, local):
    import numpy as np
    import torch
    tde = importlib.import_module("3deye_gb300")
    syn = importlib.import_module("3deye_gb300.synth")
    pl = importlib.import_module("3deye_gb300.pipeline")
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    cfg = syn.CONFIGS[WORKLOAD]
    W, K = args.warmup, args.steps
    n = W + K
    frames, traj, _ = make_frames(tde, syn, cfg, n, rank, dev)

    # CPU baseline and FP64 oracle poses (rank 0, N = 1 only), before the timed GPU passes
    cpu, f64 = None, None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        cpu, f64 = cpu_legs(cfg, frames, traj, max(1, min(args.cpu_frames, n - 1)), min(3, n - 1),
                            min(args.f64_frames, n), "640x480, 512^3")

    # ---- pass A: frames resident in HBM -----------------------------------
    # (each frame's preprocessing overlaps the previous frame's tracking on a
    # second stream; the pipeline's main stream waits for it, so the events on
    # the main stream bracket all of the K frames' work)
    p = pl.Pipeline(cfg, traj[0], use_graphs=True)
    launches = p.launches_per_frame()
    base = frames.data_ptr()
    fbytes = cfg.rows * cfg.cols * 2
    for i in range(W):
        p.enqueue(base + i * fbytes, True)
    p.sync()
    stream = torch.cuda.ExternalStream(p.stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier_sync(ws)
    clk = ClockSampler(dev).__enter__()  # runs through every GPU pass below
    time.sleep(0.05)
    with clk.window():
        e0.record(stream)
        for i in range(W, n):
            p.enqueue(base + i * fbytes, True)
        e1.record(stream)
        p.sync()
    ms = e0.elapsed_time(e1)
    ms = max_over_ranks(ws, ms)
    pose_a = p.pose()
    # distinct voxel records one raycast reads (outside the timed region):
    # as the kernel runs (empty bricks skipped) and as the reference march does
    ray_records = p.raycast_records(skip_empty=True)
    ray_records_ref = p.raycast_records(skip_empty=False)
    p.close()

    # ---- pass S: the same frames, stage by stage (serial, CUDA events) ------
    t = pl.Pipeline(cfg, traj[0], use_graphs=True, integrate_stats=True)
    for i in range(W):
        t.enqueue(base + i * fbytes, True)
    t.sync()
    t.integrate_stats(reset=True)
    t.enable_timing(K)
    for i in range(W, n):
        t.enqueue(base + i * fbytes, True)
    t.sync()
    stages = t.stage_timings(K)
    integ_ms, ray_ms = stages["integrate"], stages["raycast"]
    n_read, n_written, n_bricks = t.integrate_stats(bricks=True)
    pose_s = t.pose()
    t.close()

    # ---- pass B: end to end through the C-ABI from pinned host memory -------
    host_frames = torch.empty(frames.shape, dtype=torch.uint16, pin_memory=True)
    host_frames.copy_(frames.cpu())
    poses = torch.zeros((n, 12), dtype=torch.float64, pin_memory=True)
    status = torch.zeros(n, dtype=torch.int32, pin_memory=True)
    q = pl.Pipeline(cfg, traj[0], use_graphs=True)
    hb, pb, sb = host_frames.data_ptr(), poses.data_ptr(), status.data_ptr()
    for i in range(W):
        q.enqueue(hb + i * fbytes, False, pb + i * 96, sb + i * 4)
    q.sync()
    qs = torch.cuda.ExternalStream(q.stream)
    f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier_sync(ws)
    f0.record(qs)
    for i in range(W, n):
        q.enqueue(hb + i * fbytes, False, pb + i * 96, sb + i * 4)
    f1.record(qs)
    q.sync()
    e2e_ms = max_over_ranks(ws, f0.elapsed_time(f1))
    q.close()
    est = poses.numpy().copy()
    lost = int((status.numpy() != 0).sum())
    # overlapped (A), end-to-end (B) and serial (S) runs give the same poses
    deterministic = bool(np.array_equal(est[-1], pose_a) and np.array_equal(pose_s, pose_a))
    ate = pl.ate_rmse(est, traj)

    skip = set(x for x in args.skip.split(",") if x)
    color = export = cyclic = config1 = None
    if "color" not in skip:
        color, export = color_pass(tde, pl, torch, cfg, traj, frames, W, n, ws, dev, pose_a)
    if "cyclic" not in skip:
        cyclic = cyclic_run(tde, syn, pl, torch, dev, rank)
    if "config1" not in skip:
        config1 = config1_run(tde, syn, pl, torch, dev, rank, ws, rank == 0 and ws == 1 and not args.no_cpu_baseline)
    rgbd = None
    if "rgbd" not in skip:
        rgbd = rgbd_pass(tde, syn, torch, cfg, dev, ws, rank, rank == 0 and ws == 1 and not args.no_cpu_baseline)

    # ---- pass C: the learned refiner in place of the bilateral filter -------
    learned = None
    wpath = Path(args.refiner_weights)
    if wpath.exists() and "learned" not in skip:
        rf = importlib.import_module("3deye_gb300.refiner")
        R = rf.Refiner(1, cfg.rows, cfg.cols)
        R.set_params(np.fromfile(wpath, dtype=np.float32))
        lp = pl.Pipeline(cfg, traj[0], use_graphs=True)
        lp.set_refiner(R)
        lposes = torch.zeros((n, 12), dtype=torch.float64, pin_memory=True)
        lstat = torch.zeros(n, dtype=torch.int32, pin_memory=True)
        lb, ls = lposes.data_ptr(), lstat.data_ptr()
        for i in range(W):
            lp.enqueue(base + i * fbytes, True, lb + i * 96, ls + i * 4)
        lp.sync()
        lstream = torch.cuda.ExternalStream(lp.stream)
        g0, g1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier_sync(ws)
        g0.record(lstream)
        for i in range(W, n):
            lp.enqueue(base + i * fbytes, True, lb + i * 96, ls + i * 4)
        g1.record(lstream)
        lp.sync()
        l_ms = max_over_ranks(ws, g0.elapsed_time(g1))
        l_launches = lp.launches_per_frame()
        lp.close()
        # the refiner alone: batch-1 forward passes over the same frames, and
        # batch-16 training steps (raw frames against later frames as
        # targets: the timing does not depend on the values)
        out_mm = torch.empty((cfg.rows, cfg.cols), dtype=torch.uint16, device=dev)
        rs = torch.cuda.Stream(dev)
        for i in range(W):
            R.forward_ptr(base + i * fbytes, 1, out_mm.data_ptr(), 0, rs.cuda_stream)
        r0, r1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        rs.synchronize()
        r0.record(rs)
        for i in range(W, n):
            R.forward_ptr(base + i * fbytes, 1, out_mm.data_ptr(), 0, rs.cuda_stream)
        r1.record(rs)
        rs.synchronize()
        fwd_ms = r0.elapsed_time(r1) / K
        R.check_status()
        R.close()
        B = min(16, n // 2)
        T = rf.Refiner(B, cfg.rows, cfg.cols)
        T.set_params(np.fromfile(wpath, dtype=np.float32))
        for _ in range(3):
            T.train_step_ptr(base, base + B * fbytes, B, 1e-5, rs.cuda_stream)
        steps = 5
        r0.record(rs)
        for _ in range(steps):
            T.train_step_ptr(base, base + B * fbytes, B, 1e-5, rs.cuda_stream)
        r1.record(rs)
        rs.synchronize()
        train_ms = r0.elapsed_time(r1) / steps
        T.check_status()
        T.close()
        fwd_flops, train_flops = rf.conv_flops(cfg.rows, cfg.cols), rf.conv_flops(cfg.rows, cfg.cols, B, True)
        lest = lposes.numpy().copy()
        learned = {"value": round(ws * K / (l_ms * 1e-3), 2), "unit": "frames/s", "ms_per_step": round(l_ms / K, 5),
                   "ate_m": {"vs_ground_truth": round(pl.ate_rmse(lest, traj), 6),
                             "frames_tracking_lost": int((lstat.numpy() != 0).sum())},
                   "gpu_launches": l_launches * K, "weights": wpath.name,
                   "refiner_alone": {
                       "forward_ms_batch1": round(fwd_ms, 5),
                       "forward_tflops": round(fwd_flops / (fwd_ms * 1e-3) / 1e12, 1),
                       f"train_step_ms_batch{B}": round(train_ms, 4),
                       "train_tflops": round(train_flops / (train_ms * 1e-3) / 1e12, 1),
                       "peak_bf16_tflops": load_peaks_bf16(),
                       "note": "tensor-core convolution FLOPs (2 per multiply-add) over CUDA-event time on one "
                               "stream; training = forward + input gradients + weight gradients + AdamW"},
                   "note": "bf16 U-Net (tcgen05 implicit-GEMM convolutions) replaces the bilateral filter; "
                           "frames resident in HBM, same sequence as the plain line"}

    clk.__exit__(None, None, None)
    if rank != 0:
        return None
    hbm, peak_kind = load_peaks()
    S = 4 if cfg.tsdf_format in (0, 1) else 6
    k_int = len(integ_ms)
    int_avg_ms = float(np.mean(integ_ms)) if k_int else float("nan")
    ray_avg_ms = float(np.mean(ray_ms)) if len(ray_ms) else float("nan")
    vox_rw = (n_read + n_written) / max(k_int, 1)
    alg_bytes = S * vox_rw + 4 * cfg.rows * cfg.cols
    achieved = alg_bytes / (int_avg_ms * 1e-3) / 1e9
    traffic = load_traffic()
    int_traffic = None
    if traffic:
        cap_units = traffic["voxels_read_captured"] + traffic["voxels_written_captured"]
        int_traffic = int(traffic["dram_bytes_per_launch_captured"] * vox_rw / cap_units)
    # ICP: one launch per iteration; 48 B per pixel (current vertex + normal,
    # model vertex + normal) at the level the iteration runs on
    icp_iters = [int(x) for x in cfg.icp_iters]
    icp_launches = sum(icp_iters)
    icp_bytes = sum(48 * (cfg.cols >> l) * (cfg.rows >> l) * it for l, it in enumerate(icp_iters))
    icp_launch_ms = float(np.mean(stages["icp"])) / icp_launches
    ray_bytes = S * ray_records + 24 * cfg.rows * cfg.cols
    icp_achieved = icp_bytes / icp_launches / (icp_launch_ms * 1e-3) / 1e9
    # DRAM bytes of one cold ncu capture of a level-0 launch, scaled to the average launch by its
    # algorithmic bytes (traffic follows the pixels of the level)
    icp_cap = load_traffic("icp_traffic.json")
    icp_traffic = (int(icp_cap["dram_bytes_per_launch_captured"] * (icp_bytes / icp_launches) /
                       icp_cap["alg_bytes_captured"]) if icp_cap else None)
    fps = ws * K / (ms * 1e-3)
    line = {
        "metric": METRIC, "value": round(fps, 2), "unit": "frames/s", "n_gpus": ws, "steps": K, "warmup": W,
        "ms_per_step": round(ms / K, 5), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32 (TSDF stored f16+u16)", "data": DATA,
        "config": bench_config(ws, n),
        "e2e": {"value": round(ws * K / (e2e_ms * 1e-3), 2), "unit": "frames/s", "h2d_bytes_per_step": fbytes,
                "d2h_bytes_per_step": 96 + 4},
        "roofline": {"kernel": "icp_step_kernel (dominant: largest share of the frame)", "bound": "hbm",
                     "achieved": round(icp_achieved, 1), "peak": hbm, "peak_kind": peak_kind, "unit": "GB/s",
                     "frac": round(icp_achieved / hbm, 4), "traffic": icp_traffic,
                     "alg_bytes_per_launch": int(icp_bytes / icp_launches), "avg_launch_ms": round(icp_launch_ms, 5),
                     "launches_per_frame": icp_launches,
                     "note": "maps are L2-resident; the iteration is latency-bound (grid hand-off, totals read, 6x6 solve, association and reduction)"},
        "kernels": {
            "integrate_bricks_kernel<fp16>": {
                "bound": "hbm", "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s",
                "frac": round(achieved / hbm, 4), "traffic": int_traffic, "alg_bytes_per_launch": int(alg_bytes),
                "avg_launch_ms": round(int_avg_ms, 5),
                "voxels_read_per_launch": int(n_read / max(k_int, 1)),
                "voxels_written_per_launch": int(n_written / max(k_int, 1)),
                "bricks_swept_per_launch": int(n_bricks / max(k_int, 1)),
                "full_sweep_equivalent_gbs": round(2 * S * cfg.voxels ** 3 / (int_avg_ms * 1e-3) / 1e9, 1)},
            "raycast_kernel<fp16>": {
                "bound": "hbm", "achieved": round(ray_bytes / (ray_avg_ms * 1e-3) / 1e9, 1), "peak": hbm,
                "unit": "GB/s", "frac": round(ray_bytes / (ray_avg_ms * 1e-3) / 1e9 / hbm, 4),
                "alg_bytes_per_launch": int(ray_bytes), "avg_launch_ms": round(ray_avg_ms, 5),
                "records_read_per_launch": ray_records, "records_reference_march": ray_records_ref,
                "note": "S x distinct voxel records read (last frame) + 24 B/px of model maps"}},
        "stages_ms_per_frame": {k: round(float(np.mean(v)), 5) for k, v in stages.items()},
        "stages_note": "stage times from a serial replay with per-stage events; the headline overlaps each "
                       "frame's preprocessing with the previous frame's tracking and fusion",
        "cpu_baseline": cpu,
        "clocks": {**clk.summary(window=True),
                   "all_gpu_passes": clk.summary(window=False),
                   "note": "sampled inside the headline's timed region (window), and over every GPU pass of the run"},
        "gpu_launches": launches * K,
        "ate_m": {"vs_ground_truth": round(ate, 6), "frames_tracking_lost": lost, "deterministic": deterministic,
                  **ate_vs_fp64(pl, est, f64)},
        "learned_refine": learned,
        "color_volume": color,
        "model_export": export,
        "cyclic_volume": cyclic,
        "config1": config1,
        "rgbd_odometry": rgbd,
    }
    return line


def run_reference(args, ws, rank, local):
    """CPU implementation of the path on the host cores (rank 0 only): the
    oracle pipeline over the same sequence as the GPU arm (the CPU sensor
    renders the GPU sensor's frames bit for bit), W warm-up frames, then K
    timed frames or as many as fit the time budget.  Imports neither the
    package nor its CUDA library."""
    if rank != 0:
        return None
    syn = load_synth()
    from oracle import oracle as orc
    from oracle.pipeline import OraclePipeline
    cfg = syn.CONFIGS[WORKLOAD]
    cores = orc.set_threads(os.cpu_count() or 1)
    W, K = args.warmup, args.steps
    n = W + K
    s_scene, s_traj, s_noise = syn.seeds(0)
    scene = syn.make_scene(cfg, s_scene)
    budget_s = float(os.environ.get("TDE_REF_BUDGET_S", "150"))
    intr = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    traj = syn.make_trajectory(cfg, s_traj, n)
    frames = lambda i: orc.apply_noise(orc.render_depth(scene, traj[i], intr), s_noise, i)
    op = OraclePipeline(cfg, traj[0])
    for i in range(W):
        op.process(frames(i))
    done, t_total = 0, 0.0
    for i in range(W, n):
        d = frames(i)
        t0 = time.perf_counter()
        op.process(d)
        t_total += time.perf_counter() - t0
        done += 1
        if t_total > budget_s:
            break
    fps = done / t_total
    sample = (f"frames {W}-{W + done - 1} ({done} of the {K} timed frames, after {W} warm-up) of the 640x480 / 512^3 "
              f"sequence through the CPU oracle pipeline, {cores} OpenMP threads, {t_total:.1f} s; the reference's "
              "OpenCL kernels need a CPU OpenCL runtime absent from this host")
    return {"metric": METRIC, "value": round(fps, 4), "unit": "frames/s", "n_gpus": ws, "steps": K, "warmup": W,
            "ms_per_step": round(1e3 * t_total / done, 3), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 (TSDF stored f16+u16)", "data": DATA,
            "config": bench_config(ws, n),
            "impl": "reference",
            "cpu_baseline": {"value": round(fps, 4), "unit": "frames/s", "cores": cores, "kind": "port",
                             "sample": sample},
            "e2e": {"value": round(fps, 4), "unit": "frames/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}


def main():
    args = parse()
    ws, rank, local = dist_init(args)
    line = run_reference(args, ws, rank, local) if args.impl == "reference" else run_ours(args, ws, rank, local)
    if line is not None:
        print(json.dumps(line))
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
