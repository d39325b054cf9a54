"""The two forms of the gradient-forming forward: the rule that chooses between them
by pixels, channels and triangles, and the large launch's form at the sizes and
channel counts that the rule keeps from it."""
import pytest

from tests import test_gpu_fit as T


@pytest.mark.parametrize("pixels,channels,prims,large", [
    ((1 << 20) - 1, 8, 1000, False), (1 << 20, 8, 1000, True), (1 << 20, 8, (1 << 16) + 1, False),
    (1 << 20, 4, 1000, False), (1 << 20, 3, 1000, True), ((5 << 18) - 1, 1, 1000, False), (5 << 18, 1, 1 << 20, True),
    ((3 << 19) - 1, 16, 1000, False), (3 << 19, 16, 1000, True), (3 << 19, 32, 1000, True),
    (3 << 19, 20, 1000, False), (1 << 21, 20, 1000, True),
    (3 << 19, 9, 6143, False), (3 << 19, 9, 6144, True), ((3 << 19) - 1, 13, 1 << 20, False),
    (3 << 19, 12, 1 << 20, False), (1 << 21, 12, 1 << 20, True), (1 << 23, 12, 1000, False)])
def test_rule(pixels, channels, prims, large):
    from diffrp_gb300 import _ffi, batch, build
    build.build()
    batch._register()
    words = _ffi.size_out("drp_batch_fit_words_size", pixels, pixels * channels - 1 if channels > 1 else pixels, prims)
    assert words == (4 * pixels if large else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("tile_log2,sizes,channels,recompute,use_images", [
    (4, [(900, 601), (850, 700)], (4, 12), False, False),
    (5, [(1030, 1025)], (1, 1), False, False),
    (5, [(1060, 1020), (1040, 1030)], (9, 13), True, False),
    (4, [(1300, 1301)], (20, 20), False, True),
    (3, [(1030, 1033)], (16, 16), False, False),
    (4, [(400, 400)] * 17, (12, 10), False, False),  # walks of eight rows
])
def test_either_form(cuda_lib, monkeypatch, large, tile_log2, sizes, channels, recompute, use_images):
    from diffrp_gb300.batch import BatchRenderer
    monkeypatch.setattr(BatchRenderer, "_fit_words", lambda self: 4 * self.total_pixels if large else 0)
    T.test_large_fit_matches_forward_and_backward(cuda_lib, tile_log2, sizes, channels, recompute, use_images)
