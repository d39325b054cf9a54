"""l1_loss's gradient kept as signs: against the gradient-writing entry point
(same loss bit for bit, same gradient), with ties, NaN and infinities, and
through second derivatives and batched upstream gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pair(n, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    p, t = torch.rand(n, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    t[::5] = p[::5]
    return p, t


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 1027, 1 << 14, 2432 * 256 * 4 + 6, (1 << 23) + 1])
@pytest.mark.parametrize("up", [1.0, -0.3, 0.0, float("inf"), float("nan")])
def test_signs_equal_written_gradient(cuda_lib, n, up):
    from diffrp_gb300 import _ffi
    from diffrp_gb300.losses import l1_loss
    p, t = _pair(n)
    if n > 4:
        p[1], t[2], p[4] = float("nan"), float("inf"), float("-inf")
    loss, grad = torch.empty((), device="cuda"), torch.empty_like(p)
    ws = torch.empty(_ffi.size_out("drp_l1_loss_workspace_size", n), dtype=torch.uint8, device="cuda")
    _ffi.call("drp_l1_loss_fwd", ws.data_ptr(), ws.numel(), p.data_ptr(), t.data_ptr(), n, 1.0 / n, loss.data_ptr(),
              grad.data_ptr(), torch.cuda.current_stream().cuda_stream)
    g = torch.tensor(up, device="cuda")
    want = grad * g
    p.requires_grad_(True)
    t.requires_grad_(True)
    got = l1_loss(p, t)
    got.backward(g)
    assert torch.equal(got.detach().view(torch.int32), loss.view(torch.int32))
    torch.testing.assert_close(p.grad, want, rtol=0, atol=0, equal_nan=True)
    torch.testing.assert_close(t.grad, -want, rtol=0, atol=0, equal_nan=True)


def test_second_derivative_and_batched_upstream(cuda_lib):
    from diffrp_gb300.losses import l1_loss
    p, t = _pair(1003)
    p.requires_grad_(True)
    sign = torch.sign(p.detach() - t) / 1003
    loss = l1_loss(p, t)
    u = torch.tensor(2.0, device="cuda", requires_grad=True)
    gp, = torch.autograd.grad(loss, p, u, create_graph=True)
    gu, = torch.autograd.grad(gp, u, torch.ones_like(gp))
    assert torch.allclose(gp, 2.0 * sign, rtol=1e-6, atol=0)
    assert torch.allclose(gu, sign.sum(), rtol=1e-4, atol=1e-6)
    rows, = torch.autograd.grad(l1_loss(p, t), p, torch.tensor([1.0, -3.0], device="cuda"), is_grads_batched=True)
    assert torch.allclose(rows, torch.stack([sign, -3.0 * sign]), rtol=1e-6, atol=0)
