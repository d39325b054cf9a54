"""The backward passes by columns (launches of many pixels) against the same
pixels taken a view at a time (the per-pixel kernels): strips cut by the image's
edges, channel counts of every walk, shared and per-view vertices, derivative
lists with repeats, and NaN gradients in background pixels, which count for
nothing.  Sums in another order: within 1e-5 of the largest."""
import numpy as np
import pytest
import torch

from diffrp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _close(got, want):
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


def _views(n, res, detail=3):
    from diffrp_gb300 import nvdr as dr
    v, f = S.displaced_icosphere(detail, 0.8, 0.02, 1)
    P = S.perspective(35.0, *res, 0.1, 20.0).astype(np.float64)
    pos = np.stack([S.clip_positions(v, P @ S.view_matrix(S.lookat_pose(e)).astype(np.float64))
                    for e in S.sphere_eyes(n, 3.0, seed=2)])
    pos, tri = torch.from_numpy(pos).cuda(), torch.from_numpy(f).cuda()
    rast, db = dr.rasterize(dr.RasterizeCudaContext(), pos, tri, res)
    return pos, tri, rast, db


@pytest.mark.parametrize("C, diff, n, res, shared", [
    (3, None, 64, (91, 93), False),
    (5, None, 64, (91, 93), True),
    (6, None, 9, (250, 257), False),
    (8, None, 17, (255, 257), False),
    (10, None, 70, (83, 95), True),
    (16, None, 64, (91, 95), False),
    (4, None, 33, (250, 257), True),
    (1, None, 66, (250, 257), False),
    (5, [1, 4], 66, (250, 257), False),
    (8, [7], 66, (250, 257), True),
    (7, [3, 0, 3], 66, (250, 257), False),
    (9, "all", 66, (250, 257), False),
])
def test_interpolate_backward(cuda_lib, C, diff, n, res, shared):
    from diffrp_gb300 import nvdr as dr
    g = torch.Generator(device="cuda").manual_seed(C)
    pos, tri, rast, db = _views(n, res)
    V = pos.shape[1]
    attr = torch.randn((V, C) if shared else (n, V, C), generator=g, device="cuda")
    nd = 0 if diff is None else (C if diff == "all" else len(diff))
    go = torch.randn((n, *res, C), generator=g, device="cuda")
    gda = torch.randn((n, *res, 2 * nd), generator=g, device="cuda")
    empty = rast[..., 3] == 0
    go[empty] = float("nan")
    gda[empty] = float("nan")

    def run(lo, hi):
        a = (attr if shared else attr[lo:hi]).clone().requires_grad_(True)
        r, d = rast[lo:hi].clone().requires_grad_(True), db[lo:hi].clone().requires_grad_(True)
        out, da = dr.interpolate(a, r, tri, rast_db=d if nd else None, diff_attrs=diff)
        torch.autograd.backward([out] + ([da] if nd else []), [go[lo:hi]] + ([gda[lo:hi]] if nd else []))
        return a.grad, r.grad, d.grad

    ga, gr, gd = run(0, n)
    parts = [run(k, k + 1) for k in range(n)]
    want = sum(p[0] for p in parts) if shared else torch.cat([p[0] for p in parts])
    _close(ga, want)
    _close(gr, torch.cat([p[1] for p in parts]))
    if nd:
        _close(gd, torch.cat([p[2] for p in parts]))
    assert bool((gr[empty] == 0).all())


@pytest.mark.parametrize("n, res, shared", [(66, (250, 257), False), (513, (91, 93), False), (66, (250, 257), True)])
def test_rasterize_backward(cuda_lib, n, res, shared):
    from diffrp_gb300 import _ffi
    g = torch.Generator(device="cuda").manual_seed(n)
    pos, tri, rast, _ = _views(n, res, detail=4)
    if shared:  # every view the first one's vertices and pixels
        pos, rast = pos[:1].contiguous(), rast[:1].expand(n, -1, -1, -1).contiguous()
    V, F = pos.shape[1], len(tri)
    gr = torch.randn((n, *res, 4), generator=g, device="cuda")
    gr[rast[..., 3] == 0] = float("nan")

    def run(lo, hi):
        p = pos if shared else pos[lo:hi]
        out = torch.zeros_like(p)
        _ffi.call("drp_rasterize_bwd", p.data_ptr(), 0 if shared else V * 4, V, tri.data_ptr(), F, hi - lo, *res,
                  rast[lo:hi].data_ptr(), gr[lo:hi].data_ptr(), None, out.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
        return out

    parts = [run(k, k + 1) for k in range(n)]
    _close(run(0, n), sum(parts) if shared else torch.cat(parts))
