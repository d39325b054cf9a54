"""Images rendered without a backward (no colour image, pixel words, blends in
place) equal the differentiable forward's bit for bit: regions cut by the
image's edges, every raster tile size, channel counts with and without 128-bit
access, meshes of several items, chunks of a recomputing renderer."""
import pytest
import torch

from diffrp_gb300 import synthetic
from diffrp_gb300.batch import BatchRenderer

pytestmark = pytest.mark.gpu


def _scene(sizes, channels, tile, tpt, **kw):
    g = torch.Generator(device="cuda").manual_seed(5)
    meshes, pos, attr, items = [], [], [], []
    for m, c in enumerate(channels):
        v, f = synthetic.icosphere(2 + m, 0.8)
        v = torch.from_numpy(v).cuda()
        v = v + 0.02 * torch.randn(v.shape, generator=g, device="cuda")
        meshes.append((torch.from_numpy(f).cuda(), len(v), c))
        attr.append(torch.rand((len(v), c), generator=g, device="cuda"))
        for h, w in sizes:
            p = torch.cat([v * torch.tensor([1.1, 1.1 * w / h, 0.5], device="cuda"), torch.ones_like(v[:, :1])], 1)
            items.append((m, (h, w)))
            pos.append(p)
    r = BatchRenderer(meshes, items, tile_log2=tile, threads_per_tri=tpt, **kw)
    return r, r.pack_positions(pos), r.pack_attributes(attr)


@pytest.mark.parametrize("tile, tpt, sizes, channels", [
    (3, 0, [(1, 1), (8, 70), (33, 20)], (3,)),
    (3, 0, [(16, 32), (17, 33)], (8, 36)),
    (4, 0, [(40, 53), (15, 65), (200, 31)], (4, 5)),
    (4, 1, [(24, 24), (7, 96)], (16, 1)),
    (5, 0, [(32, 32), (9, 100), (130, 257)], (12, 7)),
    (5, 1, [(50, 50)], (8,)),
])
@pytest.mark.parametrize("chunks", [False, True])
def test_render_without_backward(tile, tpt, sizes, channels, chunks):
    kw = dict(recompute=True, chunk_pixels=2000) if chunks else {}
    r, pos, attr = _scene(sizes, channels, tile, tpt)
    want = r(pos.clone().requires_grad_(True), attr).detach()
    r2, _, _ = _scene(sizes, channels, tile, tpt, **kw)
    for _ in range(2):  # exact lists first, then fixed-depth bins
        with torch.no_grad():
            assert torch.equal(r2(pos, attr), want)
    assert torch.equal(r2(pos, attr), want)  # nothing requires a gradient
    assert want.abs().max() > 0
