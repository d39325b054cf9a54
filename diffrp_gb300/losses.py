"""Fused image losses for fitting renders to targets.

``l1_loss(pred, target)`` equals ``(pred - target).abs().mean()`` (gradient
sign(pred - target) / n, zero at exact ties, as torch's abs) but reads both
images once and keeps the gradient's signs from the same pass
(``drp_l1_loss_sign_fwd``; the gradient itself, ``drp_l1_loss_fwd``, for
tensors that do not start on 16 bytes), instead of the separate subtract / abs / mean /
sign / multiply passes of the unfused expression.
"""
import torch
from torch.autograd.forward_ad import unpack_dual
from torch.utils._python_dispatch import _get_current_dispatch_mode

from . import _ffi

__all__ = ["l1_loss"]


class _L1(torch.autograd.Function):
    @staticmethod
    def forward(ctx, pred, target):
        n = pred.numel()
        p = pred.contiguous()
        t = target.contiguous()
        scale = 1.0 / n
        loss = torch.empty((), dtype=torch.float32, device=p.device)
        ws = torch.empty(_ffi.size_out("drp_l1_loss_workspace_size", n), dtype=torch.uint8, device=p.device)
        if (p.data_ptr() | t.data_ptr()) & 15:
            kept = torch.empty_like(p)
            entry = "drp_l1_loss_fwd"
        else:
            kept = torch.empty((n + 3) // 4, dtype=torch.uint8, device=p.device)
            entry = "drp_l1_loss_sign_fwd"
        _ffi.call(entry, ws.data_ptr(), ws.numel(), p.data_ptr(), t.data_ptr(), n, scale, loss.data_ptr(),
                  kept.data_ptr(), _ffi.stream_of(p.device))
        ctx.save_for_backward(kept)
        ctx.meta = (pred.shape, scale, target.requires_grad)
        return loss

    @staticmethod
    def backward(ctx, g):
        kept, = ctx.saved_tensors
        shape, scale, target_grad = ctx.meta
        if kept.dtype != torch.uint8:
            gp = kept * g
        else:
            grad = torch.empty(shape, dtype=torch.float32, device=kept.device)
            if not _number_in_memory(g, grad):
                gp = _decode(kept, shape, scale) * g
            elif torch.is_grad_enabled():  # autograd sees the product
                gp = _signed(kept, scale, torch.ones_like(kept[:1], dtype=torch.float32), grad) * g
            else:
                gp = _signed(kept, scale, g.resolve_neg(), grad)
        return gp, (-gp if target_grad else None)


def _number_in_memory(g, grad):
    """Whether the upstream gradient is only a number that a kernel can read,
    and grad (just allocated) only memory that it can write.  Not so: under a
    dispatch mode (a trace) or a functorch transform, with a tangent, for a
    batch of gradients, a subclass or a zero without memory; those take torch's
    operators."""
    if _get_current_dispatch_mode() is not None or type(g) is not torch.Tensor:
        return False
    try:
        return bool(g.data_ptr() and grad.data_ptr()) and unpack_dual(g).tangent is None
    except RuntimeError:  # a wrapper around the tensor that has the memory
        return False


def _signed(signs, scale, upstream, grad):
    _ffi.call("drp_l1_loss_bwd", signs.data_ptr(), grad.numel(), scale, upstream.data_ptr(), grad.data_ptr(),
              _ffi.stream_of(signs.device))
    return grad


def _decode(signs, shape, scale):
    """drp_l1_loss_bwd's gradient for an upstream of one, by torch's operators."""
    bits = signs.unsqueeze(1) >> torch.arange(4, dtype=torch.uint8, device=signs.device)
    sign = (bits & 1).to(torch.float32) - ((bits >> 4) & 1).to(torch.float32)
    return sign.reshape(-1)[:shape.numel()].reshape(shape) * scale


def l1_loss(pred, target):
    """Mean absolute error between two float32 CUDA tensors of equal shape."""
    if pred.shape != target.shape or pred.dtype != torch.float32 or target.dtype != torch.float32:
        raise RuntimeError("l1_loss expects float32 tensors of the same shape")
    if not (pred.is_cuda and target.is_cuda):
        raise RuntimeError("l1_loss expects CUDA tensors")
    return _L1.apply(pred, target)
