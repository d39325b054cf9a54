"""Images for no backward, blended in place (drp_batch_render) and with the colours
apart: the same bit for bit, whichever form the launch's size would take, and on
either side of the rule."""
import pytest
import torch

from tests import test_gpu_render as T
from tests.test_gpu_fit import _renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile, tpt, sizes, channels", [
    (3, 0, [(1, 1), (8, 70), (33, 20)], (3,)),
    (3, 0, [(16, 32), (17, 33)], (8, 36)),
    (4, 0, [(40, 53), (15, 65), (200, 31)], (4, 5)),
    (4, 1, [(24, 24), (7, 96)], (16, 1)),
    (5, 0, [(32, 32), (9, 100), (130, 257)], (12, 7)),
])
@pytest.mark.parametrize("chunks", [False, True])
def test_small_launches_in_place(cuda_lib, monkeypatch, tile, tpt, sizes, channels, chunks):
    from diffrp_gb300.batch import BatchRenderer
    monkeypatch.setattr(BatchRenderer, "_blends_in_place", lambda self: True)
    T.test_render_without_backward(tile, tpt, sizes, channels, chunks)


@pytest.mark.parametrize("tile_log2,sizes,in_place", [
    (4, [(256, 767)], False), (4, [(256, 768)], True), (5, [(384, 512)], True),
    (3, [(1024, 1024)], False), (3, [(2048, 2049)], True)])
def test_either_side_of_the_rule(cuda_lib, tile_log2, sizes, in_place):
    r, pos, attr, _ = _renderer(sizes, (4, 5), tile_log2)
    assert r._blends_in_place() == in_place
    _, _, out = r.forward_buffers(pos, attr)
    with torch.no_grad():
        assert torch.equal(r(pos, attr), out)


def test_chunks_of_both_forms(cuda_lib):
    """A recomputing renderer whose chunks lie on both sides."""
    r, pos, attr, _ = _renderer([(500, 500), (40, 30)], (4, 5), 4, recompute=True)
    r._make_chunks(250000)
    assert [c.renderer._blends_in_place() for c in r._chunks] == [True, False]
    ref, _, _, _ = _renderer([(500, 500), (40, 30)], (4, 5), 4)
    assert torch.equal(r(pos, attr), ref.forward_buffers(pos, attr)[2])
