"""The two forms of the gradient-forming forward: the rule that chooses between them
by tile, pixels, channels and triangles, and the large launch's form at the sizes and
channel counts that the rule keeps from it."""
import pytest

from tests import test_gpu_fit as T


MI = 1 << 20


@pytest.mark.parametrize("tile,pixels,channels,prims,large", [
    # up to eight channels: pixels and pixels per triangle by tile
    (5, MI - 1, 8, 1000, False), (5, MI, 8, 2 * MI, True), (5, MI, 1, MI // 32, True), (5, MI, 1, MI // 32 + 1, False),
    (5, 2 * MI, 1, 2 * MI, True), (5, MI, 4, MI // 12, True), (5, MI, 5, MI // 12 + 1, False),
    (5, 5 * MI // 4, 5, MI, True), (4, MI, 4, 1, False), (4, MI, 3, MI // 64, True), (4, MI, 8, MI // 32 + 1, False),
    (4, 5 * MI // 4 - 1, 2, 1, False), (4, 3 * MI // 2, 2, MI // 32, True), (4, 3 * MI // 2, 2, MI // 32 + 1, False),
    (4, 2 * MI, 4, MI // 8, True), (4, 2 * MI, 5, MI // 8 + 1, False), (4, 2 * MI, 8, MI // 2, True),
    (3, 8 * MI, 2, 1, False), (3, 4 * MI, 4, MI // 16, True), (3, 4 * MI, 8, MI // 4, True),
    (3, 4 * MI - 1, 8, 1, False),
    # more: multiples of eight, then the others, which a coarse mesh keeps out
    (5, MI, 16, 1, True), (4, 2 * MI - 1, 16, 1, False), (4, 2 * MI, 16, 1, True), (4, 3 * MI // 2, 24, 1, True),
    (3, MI, 32, 1, True), (3, 8 * MI, 16, 1, False),
    (5, MI, 9, MI // 256, True), (5, MI, 9, MI // 256 - 1, False), (4, 5 * MI // 4, 13, MI, True),
    (5, 2 * MI - 1, 12, MI, False), (5, 2 * MI, 12, MI, True), (4, 8 * MI, 12, MI, False),
    (5, 5 * MI // 4, 20, MI, True), (4, 2 * MI, 20, MI, True), (3, 8 * MI, 20, MI, False), (3, 4 * MI, 13, MI, True)])
def test_rule(tile, pixels, channels, prims, large):
    from diffrp_gb300 import _ffi, batch, build
    build.build()
    batch._register()
    floats = pixels * channels - 1 if channels > 1 else pixels  # items of fewer channels among them
    assert _ffi.size_out("drp_batch_fit_words_size", pixels, floats, prims, tile) == (4 * pixels if large else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("tile_log2,sizes,channels,recompute,use_images", [
    (4, [(900, 601), (850, 700)], (4, 12), False, False),
    (5, [(1030, 1025)], (1, 1), False, False),
    (5, [(1060, 1020), (1040, 1030)], (9, 13), True, False),
    (4, [(1300, 1301)], (20, 20), False, True),
    (3, [(1030, 1033)], (16, 16), False, False),
    (3, [(900, 601), (850, 700)], (8, 5), False, False),
    (4, [(400, 400)] * 17, (12, 10), False, False),  # walks of eight rows
])
def test_either_form(cuda_lib, monkeypatch, large, tile_log2, sizes, channels, recompute, use_images):
    from diffrp_gb300.batch import BatchRenderer
    monkeypatch.setattr(BatchRenderer, "_fit_words", lambda self: 4 * self.total_pixels if large else 0)
    T.test_large_fit_matches_forward_and_backward(cuda_lib, tile_log2, sizes, channels, recompute, use_images)
