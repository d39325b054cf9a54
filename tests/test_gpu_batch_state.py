"""The scratch of the batching form whose size the entry points are not told or
may be told too small: the antialias state block (a flag byte and a list entry
per pixel, nothing written past them), and a workspace without room for the
large launch's pixel words (the form for small launches runs)."""
import pytest
import torch

from diffrp_gb300 import _ffi
from tests.test_gpu_fit import _renderer


def _state_bytes(pixels):
    return (256 + pixels + 255) // 256 * 256 + 4 * pixels


def test_state_size_is_the_layout_of_this_abi_version():
    from diffrp_gb300 import batch, build
    build.build()
    batch._register()
    for n in (1, 255, 1 << 16, (1 << 20) - 1, 1 << 20, 12345678):
        assert _ffi.size_out("drp_batch_aa_state_size", n) == _state_bytes(n)


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["forward", "forward_l1", "fit_l1", "forward_l1_grad",
                                   "fit_l1_plain_workspace"])
@pytest.mark.parametrize("sizes", [[(70, 90), (33, 20)], [(1000, 1101), (33, 20)]])
def test_nothing_is_written_past_the_state(cuda_lib, monkeypatch, entry, sizes):
    r, pos, attr, target = _renderer(sizes, (4, 7), 4)
    if entry == "fit_l1_plain_workspace":
        monkeypatch.setattr(r, "_fit_words", lambda: 0)
    n, scale = _state_bytes(r.total_pixels), 1.0 / r.image_floats
    state = torch.full((n + 8 * r.total_pixels,), 0xA5, dtype=torch.uint8, device="cuda")
    rast, col = r._buffers()
    img, loss = torch.empty_like(col), torch.empty((), device="cuda")
    blocks = torch.empty(r.pixel_blocks, device="cuda")
    l1 = None
    if entry == "forward_l1":
        l1 = (target, scale, torch.empty_like(col), blocks, loss)
    elif entry != "forward":
        grads = torch.empty(pos.numel() + attr.numel(), device="cuda")
        l1 = (target, scale, blocks, loss, grads[:pos.numel()].view_as(pos), grads[pos.numel():], grads)
    call = _ffi.call
    if entry == "forward_l1_grad":
        monkeypatch.setattr(_ffi, "call", lambda name, *a: call(
            "drp_batch_forward_l1_grad" if name == "drp_batch_fit_l1" else name, *a))
    r._forward_raw(pos, attr.reshape(-1), rast, col, img, l1, flags=state)
    assert int(state[:4].view(torch.int32)) > 0  # listed pixels
    assert bool((state[n:] == 0xA5).all())
    whole = entry != "fit_l1" or r._fit_words() == 0
    assert whole == (entry != "fit_l1" or r.total_pixels < 1 << 20)
    monkeypatch.undo()
    _, color, out = r.forward_buffers(pos, attr)
    assert torch.equal(img, out)
    if whole:
        assert torch.equal(col, color)
    if l1 is not None and len(l1) == 7:
        p, a = pos.clone().requires_grad_(True), attr.clone().requires_grad_(True)
        ref, _ = r.render_l1(p, a, target)
        ref.backward()
        assert torch.allclose(loss, ref, rtol=2e-6, atol=0)
        for got, want in [(l1[4], p.grad), (l1[5], a.grad)]:
            assert float((got - want).abs().max() / want.abs().max()) <= 1e-5
