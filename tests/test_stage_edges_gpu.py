"""Stage kernels at the edges of their launches and scratch."""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,rows", [(1, 1), (33, 31), (256, 4), (257, 16), (640, 480)])
def test_estimate_combined_takes_undefined_scratch_on_any_stream(cuda, tde, cols, rows):
    """The 27 sums from scratch full of ones equal those from zeroed scratch and
    the sums of the same float terms in FP64 (the model is the current map, the
    poses the identity: every residual is zero), enqueued behind unfinished work
    on a stream of the caller's."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(cols * rows)
    it = tde.Intrinsics(500.0, 500.0, (cols - 1) / 2, (rows - 1) / 2, cols, rows)
    z = 1.0 + 0.2 * torch.rand((rows, cols), device="cuda", generator=g)
    u = torch.arange(cols, device="cuda")[None, :].float()
    v = torch.arange(rows, device="cuda")[:, None].float()
    vm = torch.stack([z * (u - it.cx) / it.fx, z * (v - it.cy) / it.fy, z], -1).contiguous()
    nm = torch.randn((rows, cols, 3), device="cuda", generator=g)
    nm = (nm / nm.norm(dim=-1, keepdim=True)).contiguous()
    nm[torch.rand((rows, cols), device="cuda", generator=g) < 0.1] = torch.nan
    n = tde.lib.tde_estimate_combined_gbuf_floats(cols, rows)
    eye, t0 = tde.mat3(np.eye(3)), tde.vec3(np.zeros(3))
    out = []
    for fill in (0, 255, 255):
        s = torch.cuda.Stream()
        m = torch.full((27,), torch.nan, device="cuda")
        gbuf = torch.full((4 * n,), fill, dtype=torch.uint8, device="cuda")
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            vs = vm * 0 + 7  # the maps are written on the same stream right before
            vs.copy_(vm)
        tde.check(tde.lib.tde_estimate_combined(vs.data_ptr(), nm.data_ptr(), vs.data_ptr(), nm.data_ptr(), C.byref(eye),
                                                C.byref(t0), C.byref(eye), C.byref(t0), C.byref(it), 0.1, 0.34,
                                                gbuf.data_ptr(), m.data_ptr(), s.cuda_stream))
        s.synchronize()
        out.append(m.cpu().numpy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    p, q = vm.double().cpu().numpy().reshape(-1, 3), nm.double().cpu().numpy().reshape(-1, 3)
    ok = ~np.isnan(q[:, 0])
    J = np.concatenate([np.cross(p[ok], q[ok]), q[ok], np.zeros((ok.sum(), 1))], 1)
    A, S = J.T @ J, np.abs(J).T @ np.abs(J)
    ref = np.array([A[i, k] for i in range(6) for k in range(i, 7)])
    mag = np.array([S[i, k] for i in range(6) for k in range(i, 7)])
    # per-thread, warp and block sums of 1024 pixels in float, a cross product and a product each rounded thrice
    assert np.all(np.abs(out[0] - ref) <= 32 * 2.0 ** -24 * mag + 1e-30)


def _volume_of(fmt, f, w):
    """Packed records of float values and weights (logical order, origin 0)."""
    if fmt == 2:
        return np.concatenate([f.astype(np.float32).view(np.uint8), w.astype(np.uint16).view(np.uint8)])
    v = f.astype(np.float16).view(np.uint16) if fmt == 1 else np.trunc(f * 32767).astype(np.int16).view(np.uint16)
    return np.stack([v, w.astype(np.uint16)], -1).reshape(-1).view(np.uint8)


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("dims,origin", [((32, 40, 128), (0, 0, 0)), ((64, 300, 128), (21, 299, 5)),
                                         ((260, 33, 128), (259, 7, 127)), ((37, 31, 128), (3, 30, 64))])
@pytest.mark.parametrize("density", ["none", "one", "sparse", "every"])
def test_volume_export_of_empty_sparse_and_full_tiles(cuda, tde, orc, fmt, dims, origin, density):
    """Extract_Tsdf_Volume equals the oracle, points, weights and order, where no
    voxel, one voxel, a few and every voxel of a tile emits (alternating signs:
    three points a voxel, more than the scatter lists at once), for rows of whole
    and of odd groups, tiles of one row to 256 and shifted origins."""
    import torch
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(n + fmt)
    w = rng.integers(1, 100, n)
    f = np.full(n, 1.0)
    if density == "one":
        f[rng.integers(0, n)] = -0.5
    elif density == "sparse":
        f[rng.random(n) < 0.002] = -0.25
        f[rng.random(n) < 0.01] = 0.5
    elif density == "every":
        z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        f = np.where((x + y + z).ravel() % 2 == 0, 0.5, -0.5)
    if density == "none":
        w[:] = 0
    if density == "one":  # its neighbours emit, being neither 1 nor unseen
        f[f == 1.0] = 0.75
    vol = _volume_of(fmt, f, w)
    ob = orc.make_rb(dims, (1.0, 1.0, 1.0))
    ob.origin_GRID[:] = origin
    cell = np.array([1.0 / nx, 1.0 / ny, 1.0 / nz], np.float32)
    po, wo, no = orc.extract_tsdf_volume(vol, fmt, ob, cell, weights=True)
    assert (no == 0) == (density == "none")
    rb = tde.round_buffer(dims, (1.0, 1.0, 1.0), origin)
    dv = torch.from_numpy(vol.copy()).cuda()
    for cap in (max(no, 1), max(no // 2, 1)):
        pts, wts, k = tde.extract_tsdf_volume(dv, fmt, rb, tuple(cell), capacity=cap, weights=True)
        assert k == no
        m = min(cap, no)
        assert np.array_equal(pts.cpu().numpy()[:m].view(np.uint32), po[:m].view(np.uint32))
        assert np.array_equal(wts.cpu().numpy()[:m], wo[:m])


@pytest.mark.parametrize("cols,rows", [(2, 2), (13, 14), (33, 9), (44, 20), (45, 21), (46, 45), (97, 37)])
def test_bilateral_and_pyramid_at_window_edges(cuda, tde, orc, cols, rows):
    """Images below, at and above the size from which a block's windows stay
    inside: the filter within its rounding of the oracle's weighted mean, the
    pyramid level equal."""
    import torch
    rng = np.random.default_rng(cols * 100 + rows)
    d = (1500 + 40 * rng.random((rows, cols)) + np.arange(cols) * 2).astype(np.uint16)
    d[rng.random((rows, cols)) < 0.05] = 0
    src = torch.from_numpy(d.view(np.int16)).to("cuda").view(torch.uint16)
    out = tde.bilateral_filter(src, None, 4.5, 30.0, 32767).cpu().numpy().astype(np.float64)
    _, ratio = orc.bilateral(d, 4.5, 30.0, 32767, want_ratio=True)
    ratio = np.nan_to_num(ratio)  # a hole in the last row or column: nothing in its window counts
    # 169 additions and products a sum, weights off by up to 2 + 1.2 |x| units (|x| < 20 where they count), two sums
    tol = 2 * (2 * 169 + 26) * 2.0 ** -24
    assert np.all(np.abs(out - ratio) <= 0.5 + tol * ratio)
    lvl = tde.depth_pyramid_level(src, 30.0).cpu().numpy()
    assert np.array_equal(lvl, orc.pyramid(d, 30.0))


@pytest.mark.parametrize("voxels,fmt", [(96, 2), (96, 1), (40, 1), (52, 0)])
def test_empty_bricks_are_skipped_exactly(cuda, tde, orc, voxels, fmt):
    """The pipeline's model maps (cast with the empty bricks' masks) equal a cast
    of the same volume that skips nothing, bit for bit: while frames arrive,
    after a shift that leaves bricks across the origin, and after a restore.
    Volumes of whole super-bricks, of whole bricks, and of neither."""
    syn = importlib.import_module("3deye_gb300.synth")
    pl = importlib.import_module("3deye_gb300.pipeline")
    cfg = syn.small_config("c1", frames=8, cols=97, rows=61, voxels=voxels, fmt=fmt)
    scene, traj = syn.make_scene(cfg, 1000), syn.make_trajectory(cfg, 2000)
    intr = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    depths = [orc.apply_noise(orc.render_depth(scene, traj[i], intr), 3000, i) for i in range(cfg.frames)]
    it = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    tde.lib.tde_memcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]

    def check(p):
        import torch
        vol, rb = p.volume()
        cell = [np.float32(rb.volume_size.x) / np.float32(voxels)] * 3
        got = []
        for ptr in p.model_maps(0):
            a = np.zeros((cfg.rows, cfg.cols, 3), np.float32)
            tde.check(tde.lib.tde_memcpy(a.ctypes.data_as(C.c_void_p), C.c_void_p(ptr), a.nbytes, 1))
            got.append(a)
        pose = p.pose().astype(np.float32)
        ref = [torch.empty((cfg.rows, cfg.cols, 3), dtype=torch.float32, device=cuda) for _ in range(2)]
        R, t, cs = tde.mat3(pose[:9].reshape(3, 3)), tde.vec3(pose[9:]), tde.vec3(cell)
        tde.check(tde.lib.tde_raycast(vol, fmt, ref[0].data_ptr(), ref[1].data_ptr(), C.byref(t), C.byref(R),
                                      cfg.trunc_m, C.byref(it), C.byref(rb), C.byref(cs), None))
        torch.cuda.synchronize()
        assert np.isfinite(got[0]).any()
        for a, b in zip(got, ref):
            assert np.array_equal(a.view(np.uint32), b.cpu().numpy().view(np.uint32))

    p = pl.Pipeline(cfg, traj[0])
    for d in depths[:3]:
        p.process(d)
        check(p)
    p.shift((3, -2, 5))
    assert p.volume()[1].origin_GRID.x % 8 and p.volume()[1].origin_GRID.z % 8
    for d in depths[3:6]:
        p.process(d)
        check(p)
    q = pl.Pipeline(cfg, traj[0])
    q.restore(p.checkpoint())
    check(q)
    q.process(depths[6])
    check(q)


@pytest.mark.parametrize("cols,rows,voxels", [(1, 1, 16), (16, 17, 20), (33, 300, 64), (611, 457, 48)])
def test_integrate_takes_undefined_scratch_on_any_stream(cuda, tde, orc, cols, rows, voxels):
    """tde_integrate_tsdf_ex from scratch of zeros and of ones, enqueued on a
    stream of the caller's right behind the frame's scaling and followed by the
    raycast: the oracle's volume and maps, bit for bit."""
    import torch
    syn = importlib.import_module("3deye_gb300.synth")
    cfg = syn.small_config("c1", frames=2, cols=cols, rows=rows, voxels=voxels, fmt=1)
    scene, traj = syn.make_scene(cfg, 1000), syn.make_trajectory(cfg, 2000)
    oi = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cols, rows)
    it = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cols, rows)
    depth = orc.apply_noise(orc.render_depth(scene, traj[0], oi), 3000, 0)
    R, t = traj[0][:9].reshape(3, 3).astype(np.float32), traj[0][9:].astype(np.float32)
    ob = orc.make_rb((voxels,) * 3, (cfg.volume_m,) * 3, (3, 9, 14))
    rb = tde.round_buffer((voxels,) * 3, (cfg.volume_m,) * 3, (3, 9, 14))
    cell = np.full(3, cfg.cell, np.float32)
    ref = np.zeros(orc.volume_bytes(1, ob), np.uint8)
    for _ in range(2):
        orc.integrate(orc.scale_depth(depth, oi), ref, 1, cfg.trunc_m, np.ascontiguousarray(R.T), t, oi, cell, ob)
    vmo, nmo = orc.raycast(ref, 1, ob, oi, R, t, cfg.trunc_m, cell)
    L, V, I, F = tde.lib, C.c_void_p, C.c_int, C.c_float
    pM, pV, pI, pRB = (C.POINTER(k) for k in (tde.Matrix3f, tde.Point3f, tde.Intrinsics, tde.RoundBuffer))
    L.tde_integrate_tsdf_scratch_bytes.restype = C.c_size_t
    L.tde_integrate_tsdf_scratch_bytes.argtypes = [I, I, pRB]
    L.tde_integrate_tsdf_ex.argtypes = [V, V, I, F, pM, pV, pI, pV, pRB, I, V, C.c_size_t, V, V]
    sb = L.tde_integrate_tsdf_scratch_bytes(cols, rows, C.byref(rb))
    d = torch.from_numpy(depth.view(np.int16)).cuda()
    Ri, Rm, tt, cs = tde.mat3(R.T.copy()), tde.mat3(R), tde.vec3(t), tde.vec3(cell)
    for fill in (0, 255):
        s = torch.cuda.Stream()
        scratch = torch.full((sb,), fill, dtype=torch.uint8, device="cuda")
        vol = torch.zeros(ref.size, dtype=torch.uint8, device="cuda")
        sd = torch.empty((rows, cols), device="cuda")
        maps = torch.empty((2, rows, cols, 3), device="cuda")
        s.wait_stream(torch.cuda.current_stream())
        for _ in range(2):
            tde.check(tde.lib.tde_scale_depth(d.data_ptr(), sd.data_ptr(), C.byref(it), s.cuda_stream))
            tde.check(tde.lib.tde_integrate_tsdf_ex(sd.data_ptr(), vol.data_ptr(), 1, cfg.trunc_m, C.byref(Ri),
                                                    C.byref(tt), C.byref(it), C.byref(cs), C.byref(rb), 128,
                                                    scratch.data_ptr(), sb, None, s.cuda_stream))
        tde.check(tde.lib.tde_raycast(vol.data_ptr(), 1, maps[0].data_ptr(), maps[1].data_ptr(), C.byref(tt),
                                      C.byref(Rm), cfg.trunc_m, C.byref(it), C.byref(rb), C.byref(cs), s.cuda_stream))
        s.synchronize()
        assert np.array_equal(vol.cpu().numpy(), ref)
        got = maps.cpu().numpy()
        for a, b in zip(got, (vmo, nmo)):
            assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.nan_to_num(a), np.nan_to_num(b))


@pytest.mark.parametrize("cols,rows,levels", [(64, 32, 1), (256, 128, 1), (257, 128, 1), (330, 200, 2), (320, 240, 3)])
def test_odometry_steps_in_a_cluster_and_in_launches(cuda, tde, orc, cols, rows, levels):
    """Levels of 1, 16 (the most that one cluster takes) and 17 blocks, and a
    frame of both kinds: the first step is the oracle's, and all steps of a call
    end where the same steps one call at a time do, bit for bit."""
    import torch
    syn = importlib.import_module("3deye_gb300.synth")
    rg = importlib.import_module("3deye_gb300.rgbd")
    cfg = syn.small_config("c2", frames=2, cols=cols, rows=rows)
    scene, traj = syn.make_scene(cfg, 5), syn.make_trajectory(cfg, 5, 4)
    oi = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cols, rows)
    it = tde.Intrinsics(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cols, rows)
    host, dev = [], []
    for k in (0, 1):
        mm = np.rint(orc.render_depth(scene, traj[k], oi) * 1000).astype(np.uint16)
        rgb = orc.render_rgb(scene, traj[k], oi)
        host.append(orc.rgbd_levels(mm, rgb, levels))
        dev.append(rg.RgbdFrame(cols, rows, levels, cuda).load(torch.from_numpy(mm.view(np.int16)).to(cuda),
                                                               torch.from_numpy(rgb).to(cuda)))

    def run(iters, init):
        p = rg.default_params(levels)
        for l in range(levels):
            p.iters[l] = iters[l]
        return rg.RgbdOdometry(it, p).estimate(dev[0], dev[1], init)

    start = np.array([1, 0, 0, 0, 1, 0, 0, 0, 1, 0.002, -0.001, 0.003], np.float64)
    one = [0] * (levels - 1) + [1]
    pose, status = run(one, start)
    ref, failed = orc.rgbd_odometry(host[0], host[1], oi, one, [10.0] * levels, init_pose12=start)
    assert status == rg.STATUS_SOLVED and failed == 0
    np.testing.assert_allclose(pose, ref, rtol=0, atol=1e-7)  # the bound of the one-step test at 640x480
    steps = [3] * levels
    whole, status = run(steps, start)
    single = start
    for l in range(levels - 1, -1, -1):
        for _ in range(steps[l]):
            single, st = run([int(k == l) for k in range(levels)], single)
            assert st == rg.STATUS_SOLVED
    assert status == rg.STATUS_SOLVED and np.array_equal(whole, single)
    assert not np.array_equal(whole, pose)


def test_pose_reaches_any_host_memory(cuda, orc):
    """The pose and status of enqueued frames in pinned memory, in pinned memory
    off its alignment, and in memory that is not pinned: those of the blocking call."""
    import torch
    syn = importlib.import_module("3deye_gb300.synth")
    pl = importlib.import_module("3deye_gb300.pipeline")
    cfg = syn.small_config("c1", frames=5, cols=97, rows=61, voxels=64, fmt=2)
    scene, traj = syn.make_scene(cfg, 1000), syn.make_trajectory(cfg, 2000)
    intr = orc.Intr(cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.cols, cfg.rows)
    depths = [orc.apply_noise(orc.render_depth(scene, traj[i], intr), 3000, i) for i in range(cfg.frames)]
    p = pl.Pipeline(cfg, traj[0])
    ref = [p.process(d) for d in depths]
    p.close()
    host = torch.from_numpy(np.stack(depths).view(np.int16)).pin_memory()
    pinned = torch.full((4096,), 77, dtype=torch.uint8).pin_memory()
    plain = np.full(4096, 77, np.uint8)
    for base, off in ((pinned.data_ptr(), 0), (pinned.data_ptr(), 3), (plain.ctypes.data, 8), (plain.ctypes.data, 1)):
        p = pl.Pipeline(cfg, traj[0])
        for i in range(cfg.frames):
            p.enqueue(host[i].data_ptr(), False, base + off + 96 * i, base + 2048 + off + 4 * i)
        p.sync()
        got = (pinned.numpy() if base == pinned.data_ptr() else plain).copy()
        pose = got[off:off + 96 * cfg.frames].view(np.float64).reshape(-1, 12)
        status = got[2048 + off:2048 + off + 4 * cfg.frames].view(np.int32)
        for i, (rp, rs) in enumerate(ref):
            assert np.array_equal(pose[i], rp) and status[i] == rs
        assert (got[off + 96 * cfg.frames:2048 + off] == 77).all() and (got[2048 + off + 4 * cfg.frames:] == 77).all()
        p.close()
        pinned.fill_(77)
        plain[:] = 77
