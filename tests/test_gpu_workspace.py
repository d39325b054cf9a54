"""A renderer's workspace that grows: the old buffer is given back when only its own
stream used it, kept for captured graphs and other streams; results stay."""
import pytest
import torch

from tests.test_gpu_fit import _renderer

pytestmark = pytest.mark.gpu


def test_growing_gives_the_old_buffer_back(cuda_lib):
    r, pos, attr, target = _renderer([(1000, 1101)], (8, 8), 5)
    with torch.no_grad():
        for _ in range(3):
            out = r(pos, attr)
    small = r._wsh.buf.numel()
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    p = pos.clone().requires_grad_(True)
    _, img = r.render_l1(p, attr, target, grads_in_forward=True)
    assert r._wsh.buf.numel() > small and not r._wsh.retired
    assert torch.equal(img, out)
    del img, _, p
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - base <= r._wsh.buf.numel() - small + (1 << 21)


@pytest.mark.parametrize("how", ["graph", "stream"])
def test_growing_keeps_a_buffer_in_use_elsewhere(cuda_lib, how):
    r, pos, attr, target = _renderer([(1000, 1101)], (8, 8), 5)
    with torch.no_grad():
        for _ in range(3):
            want = r(pos, attr)
    torch.cuda.synchronize()
    if how == "graph":
        graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(graph):
            out = r(pos, attr)
    else:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(side):
            out = r(pos, attr)
        torch.cuda.current_stream().wait_stream(side)
    old = r._wsh.buf
    r.render_l1(pos.clone().requires_grad_(True), attr, target, grads_in_forward=True)
    assert len(r._wsh.retired) == 1 and r._wsh.retired[0] is old
    if how == "graph":
        out.zero_()
        graph.replay()
    assert torch.equal(out, want)
