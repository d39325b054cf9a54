"""Texture backward by groups of channels: channel counts about the groups of
four, smooth coordinates (whole warps on the same four texels, in different
repetitions of the texture and beyond its borders), odd and degenerate sizes,
against the oracle within 1e-5 of the largest component (the texel sums' order
is all that differs)."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("C", [1, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("size", [(1, 9, 14), (2, 16, 16), (2, 1, 5)])
@pytest.mark.parametrize("boundary", ["wrap", "clamp", "zero", "mirror"])
@pytest.mark.parametrize("filter_mode", ["linear", "linear-mipmap-linear"])
def test_channel_groups(cuda_lib, C, size, boundary, filter_mode):
    from diffrp_gb300 import nvdr as dr
    Nt, H, W = size
    N, h, w = 2, 21, 37
    rng = np.random.default_rng(C + H)
    tex = rng.uniform(-1, 1, (Nt, H, W, C)).astype(np.float32)
    x, y = np.meshgrid(np.linspace(-1.6, 2.7, w), np.linspace(-1.3, 2.2, h))
    uv = np.stack([np.stack([x + 0.1 * n, y - 0.07 * n], -1) for n in range(N)]).astype(np.float32)
    da = (rng.uniform(-1, 1, (N, h, w, 4)) * 2.0 ** rng.uniform(-2, 4, (N, h, w, 1)) / max(H, W)).astype(np.float32)
    gout = rng.standard_normal((N, h, w, C)).astype(np.float32)
    mipped = filter_mode != "linear"
    tex_t, uv_t = _t(tex).requires_grad_(True), _t(uv).requires_grad_(True)
    da_t = _t(da).requires_grad_(True) if mipped else None
    out = dr.texture(tex_t, uv_t, da_t, filter_mode=filter_mode, boundary_mode=boundary)
    out.backward(_t(gout))
    L = O.tex_levels(H, W) if mipped else 1
    g0, gpyr, guv, gda = O.tex_bwd(tex, O.tex_mip_build(tex, L), L, uv, da if mipped else None, gout, filter_mode,
                                   boundary)
    for got, want in [(tex_t.grad, O.tex_mip_bwd(g0, gpyr, L)), (uv_t.grad, guv)] + ([(da_t.grad, gda)] if mipped else []):
        got = got.cpu().numpy()
        assert np.abs(got - want).max() <= 1e-5 * max(np.abs(want).max(), 1e-30)
