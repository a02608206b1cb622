"""When a call of Estimate_Combined is complete."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(tde, cols, rows, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    it = tde.Intrinsics(500.0, 500.0, (cols - 1) / 2, (rows - 1) / 2, cols, rows)
    vm = torch.rand((rows, cols, 3), device="cuda", generator=g) + 0.5
    u, v = torch.arange(cols, device="cuda")[None, :], torch.arange(rows, device="cuda")[:, None]
    vm[..., 0] = vm[..., 2] * (u - it.cx) / it.fx
    vm[..., 1] = vm[..., 2] * (v - it.cy) / it.fy
    nm = torch.randn((rows, cols, 3), device="cuda", generator=g)
    nm = nm / nm.norm(dim=-1, keepdim=True)
    eye, t0 = tde.mat3(np.eye(3)), tde.vec3(np.zeros(3))
    n = tde.lib.tde_estimate_combined_gbuf_floats(cols, rows)
    gbuf = torch.empty(n, device="cuda")

    def run(m, stream):
        tde.check(tde.lib.tde_estimate_combined(vm.data_ptr(), nm.data_ptr(), vm.data_ptr(), nm.data_ptr(), C.byref(eye),
                                                C.byref(t0), C.byref(eye), C.byref(t0), C.byref(it), 0.1, 0.34,
                                                gbuf.data_ptr(), m.data_ptr(), stream.cuda_stream))

    return run, (vm, nm, gbuf)


@pytest.mark.parametrize("cols,rows", [(16, 16), (640, 480)])
def test_the_call_returns_with_its_result(cuda, tde, cols, rows):
    """Behind unfinished work on the caller's stream the sums are in place when the
    call returns: another stream reads them and writes over the scratch at once."""
    import torch
    run, keep = _call(tde, cols, rows, 3)
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    m = torch.full((27,), torch.nan, device="cuda")
    torch.cuda.synchronize()
    run(m, s)
    torch.cuda.synchronize()
    ref = m.cpu()
    assert torch.isfinite(ref).all() and ref.any()
    m.fill_(torch.nan)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)  # some 10 ms
    run(m, s)
    done = s.query()
    with torch.cuda.stream(other):
        got = m.clone()
        keep[2].fill_(torch.nan)
    torch.cuda.synchronize()
    assert done and torch.equal(got.cpu(), ref) and torch.equal(m.cpu(), ref)


def test_a_captured_call_runs_with_its_graph(cuda, tde):
    import torch
    run, _ = _call(tde, 257, 40, 4)
    s = torch.cuda.Stream()
    m = torch.full((27,), torch.nan, device="cuda")
    torch.cuda.synchronize()
    run(m, s)
    ref = m.cpu()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        run(m, s)
    m.fill_(torch.nan)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(m.cpu(), ref)
        m.fill_(torch.nan)
