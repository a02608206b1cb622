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
