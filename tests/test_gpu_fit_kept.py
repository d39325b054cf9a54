"""What render_l1(grads_in_forward=True) holds from its forward to its backward,
and that a backward through the images interpolates the colours again only where
the forward stored none."""
import pytest
import torch

from diffrp_gb300 import _ffi
from tests.test_gpu_fit import _renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,color_floats", [([(70, 90), (33, 20)], 1), ([(1000, 1101), (33, 20)], 0)])
def test_buffers_kept_and_colours_formed_again(cuda_lib, monkeypatch, sizes, color_floats):
    r, pos, attr, target = _renderer(sizes, (4, 7), 4)
    p, a = pos.clone().requires_grad_(True), attr.clone().requires_grad_(True)
    kept, names, call = {}, [], _ffi.call

    def pack(t):
        kept[t.data_ptr()] = t.numel() * t.element_size()
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        loss, img = r.render_l1(p, a, target, grads_in_forward=True)
    # inputs, target, images, gradients, rast, and the colours of a small launch
    floats = 2 * (pos.numel() + attr.numel()) + (2 + color_floats) * r.image_floats + 4 * r.total_pixels
    assert sum(kept.values()) == 4 * floats
    monkeypatch.setattr(_ffi, "call", lambda name, *x: (names.append(name), call(name, *x))[1])
    (loss + img.sum()).backward()
    assert names.count("drp_batch_colors") == (0 if color_floats else 1)
