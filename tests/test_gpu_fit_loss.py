"""The loss of the large-launch gradient-forming forward against exact sums, on
images that nothing covers (the images are zero, so the targets are the errors)."""
import pytest
import torch

from diffrp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

HW = 1024


@pytest.fixture(autouse=True)
def region_form(monkeypatch):
    from diffrp_gb300.batch import BatchRenderer
    monkeypatch.setattr(BatchRenderer, "_fit_words", lambda self: 4 * self.total_pixels)


def _loss(views, C, fill):
    from diffrp_gb300.batch import BatchRenderer
    v, f = S.icosphere(1, 0.8)
    r = BatchRenderer([(torch.from_numpy(f).cuda(), len(v), C)], [(0, (HW, HW))] * views, tile_log2=5)
    pos = torch.tensor([[0.0, 0.0, 5.0, 1.0]], device="cuda").repeat(r.pos_rows, 1)  # beyond the far plane
    target = torch.zeros(views, HW, HW, C, device="cuda")
    fill(target)
    loss, img = r.render_l1(pos.requires_grad_(True), torch.rand(len(v) * C, device="cuda"), target.reshape(-1),
                            grads_in_forward=True)
    assert not img.any()
    return float(loss.detach().double())


@pytest.mark.parametrize("views", [1, 2])
def test_sums_of_regions_keep_their_low_parts(cuda_lib, views):
    """One error of 2^24 - 1 in every region of 32 x 16 pixels: every region's sum
    and the mean are float32 numbers, sums of a few regions are not."""
    def fill(t):
        t[:, ::16, ::32, 0] = 2.0 ** 24 - 1
    assert _loss(views, 4, fill) == (2.0 ** 24 - 1) / (32 * 16 * 4)


@pytest.mark.parametrize("views", [1, 2])  # walks of four rows and of eight
@pytest.mark.parametrize("C,x", [(1, 16311569.0), (4, 3689373.0), (12, 744441.0)])
def test_equal_errors(cuda_lib, views, C, x):
    """Sums over a pixel's channels are exact here.  Roundings left (u = 2^-24 each):
    two of a compensated sum over rows, two over a region's warps, one each of the
    total, of 1 / n and of the product."""
    loss = _loss(views, C, lambda t: t.fill_(x))
    assert abs(loss - x) <= 7 * 2.0 ** -24 * x
