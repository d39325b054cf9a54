"""drp_batch_forward_l1_grad, the form of drp_batch_fit_l1 that also fills the
colour image: the same images, loss and gradients, and the ordinary forward's
colours, in a small and in a large launch."""
import pytest
import torch

from diffrp_gb300 import _ffi
from tests.test_gpu_fit import _renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, channels", [([(70, 90), (33, 20)], (8, 5)), ([(1000, 1101), (33, 20)], (4, 7))])
def test_full_colour_entry(cuda_lib, monkeypatch, sizes, channels):
    r, pos, attr, target = _renderer(sizes, channels, 4)
    _, color, out = r.forward_buffers(pos, attr)

    def run(entry):
        rast, col = r._buffers()
        img = torch.empty_like(col)
        grads = torch.empty(pos.numel() + attr.numel(), device="cuda")
        loss, blocks = torch.empty((), device="cuda"), torch.empty(r.pixel_blocks, device="cuda")
        call = _ffi.call
        monkeypatch.setattr(_ffi, "call", lambda name, *a: call(entry if name == "drp_batch_fit_l1" else name, *a))
        r._forward_raw(pos, attr.reshape(-1), rast, col, img,
                       (target, 1.0 / r.image_floats, blocks, loss, grads[:pos.numel()].view_as(pos),
                        grads[pos.numel():], grads), flags=r._flags())
        monkeypatch.undo()
        return col, img, loss, grads

    col, img, loss, grads = run("drp_batch_forward_l1_grad")
    _, img2, loss2, grads2 = run("drp_batch_fit_l1")
    assert torch.equal(col, color) and torch.equal(img, out) and torch.equal(img2, out)
    assert torch.equal(loss, loss2)
    assert float((grads - grads2).abs().max()) <= 1e-5 * float(grads.abs().max())
