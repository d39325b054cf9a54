"""The fine raster's form for launches of many tiles (128 threads per tile)
against the CPU oracle: rast, derivatives and peeling keys bit for bit, with
lists longer than one chunk of 128 primitives, empty tiles, clipped triangles,
tiles cut by the image's edges, and a list capacity that overflows."""
import numpy as np
import pytest
import torch

import oracle as O
from tests import scenes

pytestmark = pytest.mark.gpu


def _views(kind, res, n):
    if kind == "dense":
        pos, tri = scenes.random_soup(700, seed=5)  # several hundred per tile
    elif kind == "clipped":
        pos, tri = scenes.near_crossing()
    else:
        pos, tri = scenes.sphere_view(3, res=res)
    return np.stack([pos.reshape(-1, 4)] * n).astype(np.float32), tri


@pytest.mark.parametrize("tile_log2, kind, res, n", [
    (4, "dense", (200, 203), 30),
    (4, "sphere", (1111, 1130), 1),
    (4, "clipped", (137, 161), 50),
    (5, "dense", (130, 133), 500),
    (5, "sphere", (321, 350), 102),
])
def test_many_tiles(cuda_lib, tile_log2, kind, res, n):
    from diffrp_gb300 import nvdr as dr
    pos, tri = _views(kind, res, n)
    T = 1 << tile_log2
    assert n * -(-res[0] // T) * -(-res[1] // T) >= {4: 4864, 5: 12288}[tile_log2]
    r_ref, db_ref, _ = O.rasterize(pos[0], tri, res)
    pos_t = torch.from_numpy(pos).cuda()
    tri_t = torch.as_tensor(np.ascontiguousarray(tri)).cuda()
    ctx = dr.RasterizeCudaContext(tile_log2=tile_log2)
    ref = torch.from_numpy(np.asarray(r_ref)).cuda().reshape(1, *res, 4)
    ref_db = torch.from_numpy(np.asarray(db_ref)).cuda().reshape(1, *res, 4)
    for _ in range(2):  # exact lists, then fixed-depth bins
        rast, db = dr.rasterize(ctx, pos_t, tri_t, res)
        assert bool((rast == ref).all()) and bool((db == ref_db).all())
    assert float(rast[..., 3].max()) > 0
    with dr.DepthPeeler(ctx, pos_t, tri_t, res) as peeler:
        first, _ = peeler.rasterize_next_layer()
        second, _ = peeler.rasterize_next_layer()
    assert bool((first == ref).all()) and bool((second == second[:1]).all())
    small = dr.RasterizeCudaContext(tile_log2=tile_log2)
    with dr.DepthPeeler(small, pos_t[:1], tri_t, res) as peeler:  # few tiles: the other form
        peeler.rasterize_next_layer()
        want, _ = peeler.rasterize_next_layer()
    assert bool((second[:1] == want).all())
