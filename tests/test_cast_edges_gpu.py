"""The raycast right behind its volume's writer, and at the edges of its launch
and of its strides across empty bricks."""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _declare(tde):
    L, V, I, F = tde.lib, C.c_void_p, C.c_int, C.c_float
    pM, pV, pI, pRB = (C.POINTER(k) for k in (tde.Matrix3f, tde.Point3f, tde.Intrinsics, tde.RoundBuffer))
    L.tde_integrate_tsdf_scratch_bytes.restype = L.tde_brick_flags_bytes.restype = C.c_size_t
    L.tde_integrate_tsdf_scratch_bytes.argtypes = [I, I, pRB]
    L.tde_brick_flags_bytes.argtypes = [pRB]
    L.tde_integrate_tsdf_ex.argtypes = [V, V, I, F, pM, pV, pI, pV, pRB, I, V, C.c_size_t, V, V]
    L.tde_raycast_ex.argtypes = [V, I, V, V, pV, pM, F, pI, pRB, pV, V, V]
    return L


@pytest.mark.parametrize("fmt,voxels,origin", [(1, 128, (3, 126, 65)), (0, 96, (95, 1, 30)), (2, 64, (0, 0, 0))])
def test_cast_right_behind_a_sweep(cuda, tde, orc, fmt, voxels, origin):
    """Frame after frame on one stream, a sweep that lets its successor start and
    the cast of the volume and flags that it wrote, nothing between them: the
    maps and the volume of the same calls with a wait after each, bit for bit."""
    import torch
    syn = importlib.import_module("3deye_gb300.synth")
    L = _declare(tde)
    cfg = syn.small_config("c1", frames=6, cols=320, rows=240, voxels=voxels, fmt=fmt)
    scene, traj = syn.make_scene(cfg, 1000), syn.make_trajectory(cfg, 2000)
    oi = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    it = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    rb = tde.round_buffer((voxels,) * 3, (cfg.volume_m,) * 3, origin)
    cs = tde.vec3(np.full(3, cfg.cell, np.float32))
    sd = [torch.from_numpy(orc.scale_depth(orc.apply_noise(orc.render_depth(scene, traj[i], oi), 3000, i), oi)).to(cuda)
          for i in range(cfg.frames)]
    sb = L.tde_integrate_tsdf_scratch_bytes(cfg.cols, cfg.rows, C.byref(rb))

    def run(wait):
        s = torch.cuda.Stream()
        vol = tde.new_volume(fmt, rb)
        flags = torch.zeros(L.tde_brick_flags_bytes(C.byref(rb)), dtype=torch.uint8, device=cuda)
        scratch = torch.empty(sb, dtype=torch.uint8, device=cuda)
        maps = torch.full((cfg.frames, 2, 2, cfg.rows, cfg.cols, 3), 7.0, device=cuda)
        torch.cuda.synchronize()
        for i in range(cfg.frames):
            R, t = traj[i][:9].reshape(3, 3).astype(np.float32), tde.vec3(traj[i][9:].astype(np.float32))
            Ri, Rm = tde.mat3(R.T.copy()), tde.mat3(R)
            for k, f in enumerate((flags.data_ptr(), None)):  # by the flags, and without them
                tde.check(L.tde_integrate_tsdf_ex(sd[i].data_ptr(), vol.data_ptr(), fmt, cfg.trunc_m, C.byref(Ri),
                                                  C.byref(t), C.byref(it), C.byref(cs), C.byref(rb), 128,
                                                  scratch.data_ptr(), sb, flags.data_ptr(), s.cuda_stream))
                if wait:
                    s.synchronize()
                tde.check(L.tde_raycast_ex(vol.data_ptr(), fmt, maps[i, k, 0].data_ptr(), maps[i, k, 1].data_ptr(),
                                           C.byref(t), C.byref(Rm), cfg.trunc_m, C.byref(it), C.byref(rb),
                                           C.byref(cs), f, s.cuda_stream))
                if wait:
                    s.synchronize()
        s.synchronize()
        return vol.cpu().numpy(), maps.cpu().numpy()

    vol, maps = run(True)
    assert np.isfinite(maps).any() and not (maps == 7.0).any()
    for _ in range(3):
        v, m = run(False)
        assert np.array_equal(v, vol) and np.array_equal(m.view(np.uint32), maps.view(np.uint32))


# camera axes (right, down, forward) that look along each axis of the volume
LOOK = {0: [[0, 0, 1], [1, 0, 0], [0, 1, 0]], 1: [[0, 1, 0], [0, 0, 1], [1, 0, 0]], 2: [[1, 0, 0], [0, 1, 0], [0, 0, 1]]}


def _plane(dims, axis, at, toward, fmt):
    """Physical records (origin dims // 2) of a volume that is solid beyond the
    plane `at` (voxels along `axis`), seen by rays going toward +/- axis, and the
    flags of its bricks."""
    nx, ny, nz = dims
    grid = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")[2 - axis]
    f = np.clip((at - (grid + 0.5)) * toward / 4.0, -1.0, 1.0)
    for k, n in ((2, nx), (1, ny), (0, nz)):
        f = np.roll(f, n // 2, axis=k)
    w = np.full(f.size, 5, np.uint16)
    if fmt == 2:
        vol = np.concatenate([f.astype(np.float32).reshape(-1).view(np.uint8), w.view(np.uint8)])
        neg = f.astype(np.float32) < 0
    else:
        v = f.astype(np.float16) if fmt == 1 else np.trunc(f * 32767).astype(np.int16)
        vol = np.stack([v.reshape(-1).view(np.uint16), w], -1).reshape(-1).view(np.uint8)
        neg = v < 0

    def flags(e):
        out = np.zeros([-(-n // e) for n in (nz, ny, nx)], np.uint8)
        z, y, x = np.nonzero(neg)
        out[z // e, y // e, x // e] = 1
        return out.reshape(-1)

    return vol, np.concatenate([flags(8), flags(32)])


@pytest.mark.parametrize("dims", [(52, 52, 52), (49, 61, 33), (40, 72, 47), (63, 64, 17)])
@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_strides_end_where_a_short_brick_does(cuda, tde, fmt, axis, dims):
    """Axes that are not whole bricks, their origin in the middle: the last brick
    is shorter and lies inside the volume, and a surface in the voxels behind it
    is hit by the flagged cast as by the cast that skips nothing."""
    import torch
    L = _declare(tde)
    cell = np.float32(0.0625)
    rb = tde.round_buffer(dims, tuple(float(n * cell) for n in dims), tuple(n // 2 for n in dims))
    cols, rows = 24, 20
    it = tde.Intrinsics(200.0, 200.0, (cols - 1) / 2, (rows - 1) / 2, cols, rows)
    cs, trunc = tde.vec3([cell] * 3), 0.0625
    seam = dims[axis] - dims[axis] // 2  # the logical voxel that lies at physical 0
    for toward in (1, -1):
        R = np.array(LOOK[axis], np.float32)
        R = R if toward > 0 else R * np.array([-1, 1, -1], np.float32)
        t = np.array(dims, np.float32) * cell / 2
        t[axis] = (1.5 if toward > 0 else dims[axis] - 1.5) * cell
        Rm, tv = tde.mat3(R), tde.vec3(t)
        for at in np.arange(seam - 3, seam + 4, 0.7) + 0.11:  # no voxel's value is zero (then nothing is hit)
            vol, fl = _plane(dims, axis, at, toward, fmt)
            dv, df = torch.from_numpy(vol.copy()).to(cuda), torch.from_numpy(fl).to(cuda)
            assert df.numel() == L.tde_brick_flags_bytes(C.byref(rb))
            maps = torch.full((2, 2, rows, cols, 3), 7.0, device=cuda)
            torch.cuda.synchronize()
            for k, f in enumerate((None, df.data_ptr())):
                tde.check(L.tde_raycast_ex(dv.data_ptr(), fmt, maps[k, 0].data_ptr(), maps[k, 1].data_ptr(), C.byref(tv),
                                           C.byref(Rm), trunc, C.byref(it), C.byref(rb), C.byref(cs), f, None))
            torch.cuda.synchronize()
            m = maps.cpu().numpy()
            assert np.isfinite(m[0, 0]).all()
            assert np.abs(m[0, 0][..., axis] / cell - at).max() < 0.1
            assert np.array_equal(m[0].view(np.uint32), m[1].view(np.uint32)), (toward, at)


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("voxels", [52, 61])
def test_model_maps_behind_a_short_brick(cuda, tde, fmt, voxels):
    """As above by the pipeline, whose cast reads a word of flags per 32^3 bricks:
    the volume and the flags enter by a checkpoint."""
    import torch
    syn = importlib.import_module("3deye_gb300.synth")
    pl = importlib.import_module("3deye_gb300.pipeline")
    L = _declare(tde)
    L.tde_memcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    cfg = syn.small_config("c1", frames=2, cols=97, rows=61, voxels=voxels, fmt=fmt)
    it = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    p = pl.Pipeline(cfg, syn.make_trajectory(cfg, 2000)[0])
    p.shift((voxels // 2,) * 3)
    rb = p.volume()[1]
    assert (rb.origin_GRID.x, rb.origin_GRID.y, rb.origin_GRID.z) == (voxels // 2,) * 3
    cell = np.float32(rb.volume_size.x) / np.float32(voxels)
    seam = voxels - voxels // 2
    for axis in (0, 1, 2):
        for toward in (1, -1):
            R = np.array(LOOK[axis], np.float64) * (1 if toward > 0 else np.array([-1, 1, -1]))
            t = np.full(3, voxels * cell / 2, np.float64)
            t[axis] = (1.5 if toward > 0 else voxels - 1.5) * cell
            p.set_pose(np.concatenate([R.reshape(-1), t]))
            for at in np.arange(seam - 3, seam + 4, 0.7) + 0.11:
                vol, fl = _plane((voxels,) * 3, axis, at, toward, fmt)
                ck = np.array(p.checkpoint())
                ck[272:272 + vol.size] = vol  # behind the header
                ck[272 + vol.size:272 + vol.size + fl.size] = fl
                p.restore(ck)
                got = np.zeros((2, cfg.rows, cfg.cols, 3), np.float32)
                for k, ptr in enumerate(p.model_maps(0)):
                    tde.check(L.tde_memcpy(got[k].ctypes.data_as(C.c_void_p), C.c_void_p(ptr), got[k].nbytes, 1))
                ref = torch.full((2, cfg.rows, cfg.cols, 3), 7.0, device=cuda)
                torch.cuda.synchronize()
                Rm, tv, cs = tde.mat3(R.astype(np.float32)), tde.vec3(t.astype(np.float32)), tde.vec3([cell] * 3)
                tde.check(L.tde_raycast_ex(p.volume()[0], fmt, ref[0].data_ptr(), ref[1].data_ptr(), C.byref(tv),
                                           C.byref(Rm), cfg.trunc_m, C.byref(it), C.byref(rb), C.byref(cs), None, None))
                torch.cuda.synchronize()
                ref = ref.cpu().numpy()
                assert np.isfinite(ref[0]).any()
                assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), (axis, toward, at)
    p.close()


@pytest.mark.parametrize("cols,rows", [(1, 262140), (1, 262141), (2, 300001)])
def test_cast_of_a_very_tall_image(cuda, tde, cols, rows):
    """Images of more rows than a grid has blocks for (65,535 of four rows): their
    maps hold the rows of short images that look the same way."""
    import torch
    L = _declare(tde)
    n, cell = 40, np.float32(0.0625)
    vol, _ = _plane((n,) * 3, 2, 21.61, 1, 1)
    dv = torch.from_numpy(vol.copy()).to(cuda)
    rb = tde.round_buffer((n,) * 3, (float(n * cell),) * 3, (n // 2,) * 3)
    R, t, cs = tde.mat3(np.eye(3)), tde.vec3([n * cell / 2, n * cell / 2, 1.5 * cell]), tde.vec3([cell] * 3)

    def cast(first, count):
        it = tde.Intrinsics(2.0 * rows, 2.0 * rows, 0.0, float(rows // 2 - first), cols, count)
        m = torch.full((2, count, cols, 3), 7.0, device=cuda)
        torch.cuda.synchronize()
        tde.check(L.tde_raycast_ex(dv.data_ptr(), 1, m[0].data_ptr(), m[1].data_ptr(), C.byref(t), C.byref(R), 0.0625,
                                   C.byref(it), C.byref(rb), C.byref(cs), None, None))
        torch.cuda.synchronize()
        return m.cpu().numpy()

    tall = cast(0, rows)
    assert np.isfinite(tall[0]).all()
    for first in (0, rows // 2, 262140 - 37, rows - 64):
        count = min(64, rows - first)
        assert np.array_equal(tall[:, first:first + count].view(np.uint32), cast(first, count).view(np.uint32))
