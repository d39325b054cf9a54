"""Fused image losses for fitting renders to targets.

``l1_loss(pred, target)`` equals ``(pred - target).abs().mean()`` (gradient
sign(pred - target) / n, zero at exact ties, as torch's abs) but reads both
images once and keeps the gradient's signs from the same pass
(``drp_l1_loss_sign_fwd``; the gradient itself, ``drp_l1_loss_fwd``, for
tensors that do not start on 16 bytes), instead of the separate subtract / abs / mean /
sign / multiply passes of the unfused expression.
"""
import torch

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
        elif torch.is_grad_enabled() or not torch._C._has_storage(g):
            # the gradient as a tensor of its own: autograd and vmap see the product
            gp = _signed(kept, shape, scale, torch.ones_like(kept[:1], dtype=torch.float32)) * g
        else:
            gp = _signed(kept, shape, scale, g.resolve_neg())
        return gp, (-gp if target_grad else None)


def _signed(signs, shape, scale, upstream):
    grad = torch.empty(shape, dtype=torch.float32, device=signs.device)
    _ffi.call("drp_l1_loss_bwd", signs.data_ptr(), grad.numel(), scale, upstream.data_ptr(), grad.data_ptr(),
              _ffi.stream_of(signs.device))
    return grad


def l1_loss(pred, target):
    """Mean absolute error between two float32 CUDA tensors of equal shape."""
    if pred.shape != target.shape or pred.dtype != torch.float32 or target.dtype != torch.float32:
        raise RuntimeError("l1_loss expects float32 tensors of the same shape")
    if not (pred.is_cuda and target.is_cuda):
        raise RuntimeError("l1_loss expects CUDA tensors")
    return _L1.apply(pred, target)
