"""l1_loss's backward with upstream gradients that are more than a number in
memory: a tangent of its own (forward over reverse), a zero that has no memory,
a functorch level, a negated view, and an operator trace."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

pytestmark = pytest.mark.gpu

N = 1003


@pytest.fixture()
def case(cuda_lib):
    from diffrp_gb300.losses import l1_loss
    g = torch.Generator(device="cuda").manual_seed(4)
    p, t = torch.rand(N, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g)
    t[::5] = p[::5]
    want = torch.sign(p - t) * torch.tensor(1.0 / N, device="cuda")
    p.requires_grad_(True)
    return p, l1_loss(p, t), want


def _grad(loss, p, u):
    return torch.autograd.grad(loss, p, u, retain_graph=True)[0]


def test_tangent_of_the_upstream_gradient(case):
    p, loss, want = case
    with fwd.dual_level():
        u = fwd.make_dual(torch.tensor(2.0, device="cuda"), torch.tensor(-3.0, device="cuda"))
        got = fwd.unpack_dual(_grad(loss, p, u))
        assert got.tangent is not None
        torch.testing.assert_close(got.primal, 2.0 * want, rtol=1e-6, atol=0)
        torch.testing.assert_close(got.tangent, -3.0 * want, rtol=1e-6, atol=0)


def test_zero_without_memory(case):
    p, loss, want = case
    got = _grad(loss, p, torch._efficientzerotensor((), device="cuda"))
    assert torch.equal(got + torch.zeros_like(want), torch.zeros_like(want))


@pytest.mark.parametrize("transform", ["vmap", "jvp", "neg"])
def test_wrapped_upstream(case, transform):
    p, loss, want = case
    if transform == "vmap":
        got = torch.func.vmap(lambda u: _grad(loss, p, u))(torch.tensor([1.0, -3.0], device="cuda"))
        ref = torch.stack([want, -3.0 * want])
    elif transform == "jvp":
        one = torch.tensor(2.0, device="cuda")
        got, tan = torch.func.jvp(lambda u: _grad(loss, p, u), (one,), (3.0 * torch.ones_like(one),))
        torch.testing.assert_close(tan, 3.0 * want, rtol=1e-6, atol=0)
        ref = 2.0 * want
    else:
        got, ref = _grad(loss, p, torch._neg_view(torch.tensor(2.0, device="cuda"))), -2.0 * want
    torch.testing.assert_close(got, ref, rtol=1e-6, atol=0)


def test_operators_are_seen(case):
    """A dispatch mode sees the product with the upstream gradient (what a trace
    of the backward records)."""
    from torch.utils._python_dispatch import TorchDispatchMode
    p, loss, want = case

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            hit = any(a is u for a in args)
            seen.append(func) if hit and func.overloadpacket is torch.ops.aten.mul else None
            return func(*args, **(kwargs or {}))

    seen, u = [], torch.tensor(2.0, device="cuda")
    with Seen():
        got = _grad(loss, p, u)
    assert seen
    torch.testing.assert_close(got, 2.0 * want, rtol=1e-6, atol=0)
