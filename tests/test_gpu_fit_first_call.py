"""The first gradient-forming forward of a renderer whose tile lists outgrow
their first size (a few large triangles over many tiles): its gradients against
the ordinary backward's, with stored buffers and recomputing in chunks, where
the later chunks add into buffers that the first one zeroed."""
import numpy as np
import pytest
import torch

from diffrp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("tile_log2,hw", [(3, (401, 390)), (4, (1040, 1030))])  # per-pixel and region form
def test_first_call_with_overflowing_lists(cuda_lib, monkeypatch, recompute, tile_log2, hw):
    from diffrp_gb300.batch import BatchRenderer
    monkeypatch.setattr(BatchRenderer, "_fit_words",
                        lambda self: 4 * self.total_pixels if self.total_pixels >= 1 << 20 else 0)
    v, f = S.icosphere(1, 0.8)
    rng = np.random.default_rng(0)
    pos = []
    for k in range(3):
        mvp = S.perspective(40.0, hw[0], hw[1], 0.1, 20.0).astype(np.float64) @ \
            S.view_matrix(S.lookat_pose(S.sphere_eyes(1, 2.6, seed=k)[0])).astype(np.float64)
        pos.append(torch.from_numpy(S.clip_positions(v, mvp)).cuda())
    attr = torch.from_numpy(rng.uniform(0, 1, (len(v), 4)).astype(np.float32)).cuda().reshape(-1)

    def run(eager):  # a new renderer: its first forward
        r = BatchRenderer([(torch.from_numpy(f).cuda(), len(v), 4)], [(0, hw)] * 3, tile_log2=tile_log2,
                          recompute=recompute, chunk_pixels=hw[0] * hw[1])
        g = torch.Generator(device="cuda").manual_seed(5)
        target = torch.rand(r.image_floats, device="cuda", generator=g)
        p, a = r.pack_positions(pos).requires_grad_(True), attr.clone().requires_grad_(True)
        loss, img = r.render_l1(p, a, target, grads_in_forward=eager)
        loss.backward()
        for c in [c.renderer for c in r._chunks] if recompute else [r]:
            assert c.last_list_entries > 4 * c.total_prims + 4096
        return loss.detach(), img.detach(), p.grad, a.grad

    le, ime, gpe, gae = run(True)
    lr, imr, gpr, gar = run(False)
    assert torch.equal(ime, imr)
    assert torch.allclose(le, lr, rtol=2e-6, atol=0)
    for got, ref in [(gpe, gpr), (gae, gar)]:
        assert float((got - ref).abs().max() / ref.abs().max()) <= 1e-5
