"""The listed pixels' backward (those a blending pair touches) by channel count
and alignment: several channels to a lane where rows allow 16-byte access, one
otherwise (here also because an earlier mesh's attributes end off 16 bytes),
against the drop-in ops item by item: within 1e-4 of the largest, the bar of the
gradients against the float64 oracle."""
import numpy as np
import pytest
import torch

from diffrp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [(8, 8), (5, 8), (12, 16), (4, 20), (3, 32), (7, 12)])
def test_listed_pixels(cuda_lib, channels):
    from diffrp_gb300 import nvdr as dr
    from diffrp_gb300.batch import BatchRenderer
    rng = np.random.default_rng(sum(channels))
    meshes = [S.displaced_icosphere(2, 0.8, 0.05, 1), S.random_displaced_grid(7, seed=2, sigma=0.05)]
    sizes = [(70, 61), (40, 97)]
    tris = [torch.from_numpy(f).cuda() for _, f in meshes]
    r = BatchRenderer([(t, len(v), c) for t, (v, _), c in zip(tris, meshes, channels)], list(enumerate(sizes)))
    pos = []
    for k, (h, w) in enumerate(sizes):
        mvp = S.perspective(40.0, h, w, 0.1, 20.0).astype(np.float64) @ \
            S.view_matrix(S.lookat_pose(S.sphere_eyes(1, 2.6, seed=k)[0])).astype(np.float64)
        pos.append(torch.from_numpy(S.clip_positions(meshes[k][0], mvp)).cuda())
    attr = [torch.from_numpy(rng.uniform(0, 1, (len(v), c)).astype(np.float32)).cuda()
            for (v, _), c in zip(meshes, channels)]
    gout = torch.from_numpy(rng.standard_normal(r.image_floats).astype(np.float32)).cuda()
    P, A = r.pack_positions(pos).requires_grad_(True), r.pack_attributes(attr).requires_grad_(True)
    out = r(P, A)
    out.backward(gout)
    want_p, want_a = [], []
    for k, hw in enumerate(sizes):
        p, a = pos[k][None].clone().requires_grad_(True), attr[k].clone().requires_grad_(True)
        rast, _ = dr.rasterize(dr.RasterizeCudaContext(), p, tris[k], hw, grad_db=False)
        color, _ = dr.interpolate(a[None], rast, tris[k])
        img = dr.antialias(color, rast, p, tris[k])
        assert torch.equal(img[0], r.images(out)[k])
        assert not torch.equal(img, color)  # some pixels blend
        img.backward(r.images(gout)[k][None])
        want_p.append(p.grad.reshape(-1, 4))
        want_a.append(a.grad.reshape(-1))
    for got, want in [(P.grad, torch.cat(want_p)), (A.grad, torch.cat(want_a))]:
        assert float((got - want).abs().max()) <= 1e-4 * float(want.abs().max())
