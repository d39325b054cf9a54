"""Forms that only launches of 2^20 pixels and more take: the images without a
backward (four rows per warp), the colours formed again, and the sign of the loss's
gradient at ties, NaN and infinities."""
import pytest
import torch

from diffrp_gb300 import _ffi
from tests.test_gpu_fit import _renderer

pytestmark = pytest.mark.gpu

SIZES = [(1000, 1101), (33, 20)]


@pytest.mark.parametrize("tile_log2,channels", [(3, (4, 3)), (4, (8, 4)), (5, (5, 8)), (5, (40, 1))])
def test_images_without_a_backward(cuda_lib, tile_log2, channels):
    r, pos, attr, _ = _renderer(SIZES if tile_log2 > 3 else [(2049, 2048)], channels, tile_log2)
    _, _, out = r.forward_buffers(pos, attr)
    with torch.no_grad():
        assert torch.equal(r(pos, attr), out)


@pytest.mark.parametrize("sizes", [SIZES, [(70, 90), (33, 20)]])
@pytest.mark.parametrize("channels", [(8, 5), (3, 4)])
def test_colours_formed_again(cuda_lib, sizes, channels):
    r, pos, attr, _ = _renderer(sizes, channels, 4)
    rast, color, _ = r.forward_buffers(pos, attr)
    got = torch.full_like(color, float("nan"))
    _ffi.call("drp_batch_colors", r._items_dev.data_ptr(), len(r.items), r._xmap.data_ptr(), r.pixel_blocks,
              r.tri.data_ptr(), attr.data_ptr(), rast.data_ptr(), got.data_ptr(), _ffi.stream_of(attr.device))
    assert torch.equal(got, color)


@pytest.mark.parametrize("channels", [(8, 4), (3, 5), (12, 8)])
def test_gradient_at_ties_nan_and_infinities(cuda_lib, monkeypatch, channels):
    r, pos, attr, target = _renderer(SIZES, channels, 4)
    monkeypatch.setattr(r, "_fit_words", lambda: 4 * r.total_pixels)
    p, a = pos.clone().requires_grad_(True), attr.clone().requires_grad_(True)
    img = r(p, a)
    target = target.clone()
    target[::4] = img.detach()[::4]
    target[1::97], target[2::89], target[3::83] = float("nan"), float("inf"), float("-inf")
    sign = torch.sign(img.detach() - target).nan_to_num(nan=0.0)
    img.backward(sign / r.image_floats)
    q, b = pos.clone().requires_grad_(True), attr.clone().requires_grad_(True)
    loss, out = r.render_l1(q, b, target, grads_in_forward=True)
    loss.backward()
    assert torch.equal(out, img) and torch.isnan(loss)
    for got, ref in [(q.grad, p.grad), (b.grad, a.grad)]:
        assert float((got - ref).abs().max() / ref.abs().max()) <= 1e-5
