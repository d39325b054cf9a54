"""The fine raster on both sides of its rule for launches of many tiles (fewer
than 64 triangles of the mesh per tile: 128 threads per tile): the same images
bit for bit as one view at a time, which is a launch of few tiles."""
import numpy as np
import pytest
import torch

from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("triangles", [64 * 169 - 1, 64 * 169])
def test_either_side_equals_single_views(cuda_lib, triangles):
    from diffrp_gb300 import nvdr as dr
    from diffrp_gb300.batch import BatchRenderer
    res, n = (200, 203), 30  # 13 x 13 tiles of 16 pixels a view, 5070 in all
    pos, tri = scenes.random_soup(triangles, seed=5)
    pos = torch.from_numpy(np.asarray(pos, np.float32).reshape(-1, 4)).cuda()
    tri = torch.as_tensor(np.ascontiguousarray(tri)).cuda()
    views = torch.stack([pos * torch.tensor([1.0, 1.0 - 0.01 * k, 1.0, 1.0], device="cuda") for k in range(n)])
    ctx = dr.RasterizeCudaContext(tile_log2=4)
    many, _ = dr.rasterize(ctx, views, tri, res, grad_db=False)
    r = BatchRenderer([(tri, len(pos), 4)], [(0, res)] * n, tile_log2=4)
    batch, _, _ = r.forward_buffers(views.reshape(-1, 4), torch.rand(len(pos) * 4, device="cuda"))
    for k, got in enumerate(r.rast_views(batch)):
        want, _ = dr.rasterize(ctx, views[k:k + 1].contiguous(), tri, res, grad_db=False)
        assert torch.equal(many[k], want[0]) and torch.equal(got, want[0])
