"""The antialias forward by regions (from 2^17 pixels on) against the CPU
oracle: images cut inside a region (odd widths and heights, one column, one
row), several views, channel counts and alignments with and without 128-bit
copies and blends, with a soup (every edge a silhouette) and a closed mesh.
Bit for bit, as the forward is specified.  The pixel list it writes: the backward
that walks it equals the backward that evaluates every pixel (colour gradient bit
for bit, position gradient up to the order of the atomics)."""
import numpy as np
import pytest
import torch

import oracle as O
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res, C, soup, offset", [
    ((363, 365), 3, False, 0),
    ((512, 256), 4, True, 0),
    ((257, 513), 5, True, 0),
    ((260, 516), 8, False, 0),
    ((260, 516), 8, True, 1),  # colours not on 16 bytes
    ((301, 436), 1, False, 0),
    ((8, 16384), 2, True, 0),
    ((16384, 9), 3, True, 0),
    ((370, 356), 12, False, 0),
])
def test_antialias_regions(cuda_lib, res, C, soup, offset):
    from diffrp_gb300 import _ffi
    from diffrp_gb300 import nvdr as dr
    H, W = res
    assert 2 * H * W >= 1 << 17
    pos, tri = scenes.random_soup(150, seed=2) if soup else scenes.sphere_view(3, res=res)
    rng = np.random.default_rng(4)
    pos_t = torch.as_tensor(np.ascontiguousarray(pos)).cuda()
    tri_t = torch.as_tensor(np.ascontiguousarray(tri)).cuda()
    rast, _ = dr.rasterize(dr.RasterizeCudaContext(), pos_t, tri_t, res)
    rast = torch.cat([rast, rast.flip(2)])  # a second view: the mirrored ids on the same positions
    B = 2
    color = rng.uniform(0, 1, (B, H, W, C)).astype(np.float32)
    flat = torch.empty(color.size + offset, device="cuda")[offset:]
    flat.copy_(torch.from_numpy(color).cuda().reshape(-1))
    col = flat.view(B, H, W, C)
    pos2 = pos_t.reshape(1, -1, 4).expand(2, -1, -1).contiguous()
    nbr = dr.antialias_construct_topology_hash(tri_t)
    F, V = len(tri), pos2.shape[1]
    ws = torch.empty(_ffi.size_out("drp_antialias_workspace_size", B, F), dtype=torch.uint8, device="cuda")
    state = torch.empty(_ffi.size_out("drp_antialias_state_size", B, H, W), dtype=torch.uint8, device="cuda")
    out = torch.empty_like(col)
    sp = torch.cuda.current_stream().cuda_stream
    common = (col.data_ptr(), C, rast.data_ptr(), pos2.data_ptr(), V * 4, V, tri_t.data_ptr(), F, nbr.data_ptr(),
              B, H, W)
    _ffi.call("drp_antialias_fwd", ws.data_ptr(), ws.numel(), *common, out.data_ptr(), state.data_ptr(), sp)
    ref = O.antialias(color, rast.cpu().numpy(), pos2.cpu().numpy(), tri)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    assert (ref != color).any()
    go = torch.from_numpy(rng.standard_normal(ref.shape).astype(np.float32)).cuda()
    grads = []
    for st in (None, state.data_ptr()):
        gc, gp = torch.empty_like(go), torch.zeros_like(pos2)
        _ffi.call("drp_antialias_bwd", ws.data_ptr(), ws.numel(), *common, go.data_ptr(), 1.0, gc.data_ptr(),
                  gp.data_ptr(), st, sp)
        grads.append((gc, gp))
    assert torch.equal(grads[0][0], grads[1][0])
    scale = float(grads[0][1].abs().max())
    assert scale > 0 and float((grads[0][1] - grads[1][1]).abs().max()) <= 1e-5 * scale
