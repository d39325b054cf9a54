"""Dense tiles in the pixel-parallel fine raster (long lists whose small
triangles go by thread) against the CPU oracle: rast and derivatives bit for
bit; a second depth layer against the thread-per-triangle raster; lists that
overflow their capacity; small triangles beside large and clipped ones."""
import numpy as np
import pytest
import torch

import oracle as O
from diffrp_gb300 import synthetic as S
from tests import scenes

pytestmark = pytest.mark.gpu


def _mesh(n, extra, seed):
    v, f = S.random_displaced_grid(n, seed=seed, sigma=0.02)
    pos = np.concatenate([v * np.float32([0.9, 0.9, 0.3]), np.ones((len(v), 1), np.float32)], 1)
    if extra == "large":
        p2, f2 = scenes.random_soup(40, seed=seed)
    elif extra == "clipped":
        p2, f2 = scenes.near_crossing()
    else:
        return pos.astype(np.float32), f.astype(np.int32)
    return (np.concatenate([pos, p2.reshape(-1, 4)]).astype(np.float32),
            np.concatenate([f, f2 + len(pos)]).astype(np.int32))


@pytest.mark.parametrize("tile_log2", [3, 4, 5])
@pytest.mark.parametrize("n, extra, res, capacity", [
    (60, None, (33, 31), None),     # around one chunk per tile
    (200, None, (64, 50), None),    # many chunks, every triangle small
    (150, "large", (70, 96), None),
    (120, "clipped", (40, 65), None),
    (120, "large", (40, 65), 64),   # lists overflow: every tile scans all
    (24, None, (45, 45), None),     # boxes about the small limit
])
def test_dense_tiles(cuda_lib, tile_log2, n, extra, res, capacity):
    from diffrp_gb300 import nvdr as dr
    pos, tri = _mesh(n, extra, 7)
    r_ref, db_ref, _ = O.rasterize(pos, tri, res)
    pos_t, tri_t = torch.from_numpy(pos).cuda(), torch.from_numpy(tri).cuda()
    ctx = dr.RasterizeCudaContext(tile_log2=tile_log2)
    if capacity:
        ctx.ensure_capacity(capacity)
    for _ in range(2):  # exact lists, then fixed-depth bins
        rast, db = dr.rasterize(ctx, pos_t, tri_t, res)
        np.testing.assert_array_equal(rast.cpu().numpy().reshape(np.shape(r_ref)), r_ref)
        np.testing.assert_array_equal(db.cpu().numpy().reshape(np.shape(db_ref)), db_ref)
    assert (r_ref[..., 3] > 0).any()
    layers = []
    for c in (ctx, dr.RasterizeCudaContext(tile_log2=tile_log2, threads_per_tri=1)):
        with dr.DepthPeeler(c, pos_t, tri_t, res) as peeler:
            layers.append([peeler.rasterize_next_layer()[0] for _ in range(2)])
    assert torch.equal(layers[0][0], layers[1][0]) and torch.equal(layers[0][1], layers[1][1])
