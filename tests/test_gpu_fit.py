"""The large-launch form of the gradient-forming forward (render_l1 with
grads_in_forward=True from 2^20 pixels on): images, loss and gradients against
the ordinary forward and backward of the same renderer, at ragged resolutions
(columns past the image, a last region of a few rows), every raster tile size,
and channel counts that take its different loops (sums held over rows, or
per row; with and without 128-bit access)."""
import numpy as np
import pytest
import torch

from diffrp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _renderer(sizes, channels, tile_log2, recompute=False, detail=4):
    from diffrp_gb300.batch import BatchRenderer
    rng = np.random.default_rng(3)
    ico = S.displaced_icosphere(detail, 0.8, 0.02, 1)
    grid = S.random_displaced_grid(90, seed=2, sigma=0.02)  # triangles of a few pixels, open borders
    meshes = [(v, f, c) for (v, f), c in zip([ico, grid], channels)]
    items = [(k % 2, hw) for k, hw in enumerate(sizes)]
    pos = []
    for k, (m, (h, w)) in enumerate(items):
        mvp = S.perspective(40.0, h, w, 0.1, 20.0).astype(np.float64) @ \
            S.view_matrix(S.lookat_pose(S.sphere_eyes(1, 2.6, seed=k)[0])).astype(np.float64)
        pos.append(torch.from_numpy(S.clip_positions(meshes[m][0], mvp)).cuda())
    r = BatchRenderer([(torch.from_numpy(f).cuda(), len(v), c) for v, f, c in meshes], items, tile_log2=tile_log2,
                      recompute=recompute, chunk_pixels=1 << 20 if recompute else 1 << 23)
    attr = r.pack_attributes([torch.from_numpy(rng.uniform(0, 1, (len(v), c)).astype(np.float32)).cuda()
                              for v, _, c in meshes])
    target = torch.from_numpy(rng.uniform(0, 1, r.image_floats).astype(np.float32)).cuda()
    return r, r.pack_positions(pos), attr, target


@pytest.mark.parametrize("tile_log2,sizes,channels,recompute,use_images", [
    (5, [(1000, 1101), (33, 20)], (8, 4), False, False),
    (5, [(1030, 1025)], (8, 8), False, True),
    (4, [(900, 601), (850, 700)], (4, 12), False, False),
    (4, [(1030, 1033)], (3, 3), False, False),
    (3, [(900, 601), (850, 700)], (8, 5), False, False),
    (4, [(400, 400)] * 17, (8, 4), False, True),  # from 4096 regions on: taller walks
    (5, [(1060, 1020), (1040, 1030)], (8, 13), True, False),
])
def test_large_fit_matches_forward_and_backward(cuda_lib, tile_log2, sizes, channels, recompute, use_images):
    r, pos, attr, target = _renderer(sizes, channels, tile_log2, recompute)
    assert r.total_pixels >= 1 << 20
    w = torch.linspace(-1, 1, r.image_floats, device="cuda")

    def run(eager):
        p, a = pos.clone().requires_grad_(True), attr.clone().requires_grad_(True)
        loss, img = r.render_l1(p, a, target, grads_in_forward=eager)
        (3.0 * loss + ((img * w).sum() if use_images else 0.0)).backward()
        return loss.detach(), img.detach(), p.grad, a.grad

    le, ime, gpe, gae = run(True)
    lr, imr, gpr, gar = run(False)
    assert torch.equal(ime, imr)
    assert torch.allclose(le, lr, rtol=2e-6, atol=0)
    for got, ref in [(gpe, gpr), (gae, gar)]:
        assert float((got - ref).abs().max() / ref.abs().max()) <= 1e-5
    le2 = run(True)[0]
    assert torch.equal(le, le2)  # fixed-order sums
