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
