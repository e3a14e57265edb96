"""Training-mode BatchNorm with the residual add and ReLU behind it
(``csrc/kernels/batchnorm.cu``), for channels-last activations.

torch runs BatchNorm, the add and the ReLU as separate passes over the
activations in both directions.  Here the forward is two passes (statistics,
then everything else) and the backward two (the channel sums, then ``dx``); the
ReLU's mask is recomputed from the input instead of being read back.
"""

from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _C
from ._plain import native, ordinary, plain_module


class _BatchNormActFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, residual, weight, bias, running_mean, running_var, tracked, momentum, eps, relu, twice):
        y, mean, rstd = _C.batch_norm_fwd(x, residual, weight, bias, running_mean, running_var, tracked, momentum,
                                          eps, relu)
        torch.autograd.graph.increment_version(tracked)  # as torch's own layer does, which adds 1 in place
        ctx.relu, ctx.eps, ctx.has_residual = relu, eps, residual is not None
        ctx.save_for_backward(x, weight, bias, mean, rstd, y if relu and residual is not None else None)
        if not twice:
            return y
        ctx.set_materialize_grads(False)  # an unused output arrives as None, not as zeros
        return y, y.view_as(y)

    @staticmethod
    def backward(ctx, dy, dy2=None):
        if dy is None:
            dy, dy2 = dy2, None
        if dy is None:
            return (None,) * 11
        x, weight, bias, mean, rstd, y = ctx.saved_tensors
        if torch.is_grad_enabled():  # the graph of this backward is wanted: torch's own ops have one
            dy = dy if dy2 is None else dy + dy2
            out = F.batch_norm(x, None, None, weight, bias, True, 0.0, ctx.eps)
            if ctx.relu:
                dy = torch.where((out if y is None else y).detach() <= 0, torch.zeros_like(dy), dy)
            inputs = (x, weight, bias)
            grads = iter(torch.autograd.grad(out, [t for t in inputs if t.requires_grad], dy, create_graph=True)
                         if any(t.requires_grad for t in inputs) else ())
            dx, dgamma, dbeta = (next(grads) if t.requires_grad else None for t in inputs)
            return dx, dy if ctx.has_residual else None, dgamma, dbeta, None, None, None, None, None, None, None
        # Saved-tensor hooks may have brought x and y back in another layout (save_on_cpu with pinned memory).
        x, dy = (t.contiguous(memory_format=torch.channels_last) for t in (x, dy))
        y = None if y is None else y.contiguous(memory_format=torch.channels_last)
        if dy2 is not None:
            dy2 = dy2.contiguous(memory_format=torch.channels_last)
            if y is None:
                dy, dy2 = dy + dy2, None
        dx, dres, dgamma, dbeta = _C.batch_norm_bwd(dy, x, y, weight, bias, mean, rstd, ctx.relu, dy2)
        if ctx.has_residual and not ctx.relu:
            dres = dy
        return dx, dres if ctx.has_residual else None, dgamma, dbeta, None, None, None, None, None, None, None


def _channels_last(t: torch.Tensor) -> bool:
    return t.is_contiguous(memory_format=torch.channels_last) and t.data_ptr() % 16 == 0


def _fusable(bn: nn.BatchNorm2d, x: torch.Tensor, residual: torch.Tensor | None) -> bool:
    if not (native(x) and bn.training and plain_module(bn, nn.BatchNorm2d) and x.dim() == 4):
        return False
    c = x.shape[1]
    params = (bn.weight, bn.bias, bn.running_mean, bn.running_var)
    if bn.momentum is None or bn.num_batches_tracked is None or any(
            p is None or not ordinary(p) or p.dtype != torch.float32 or p.device != x.device or p.numel() != c or not p.is_contiguous()
            or p.data_ptr() % 16 for p in params):
        return False
    if bn.num_batches_tracked.device != x.device or bn.num_batches_tracked.dtype != torch.long:
        return False
    if x.dtype not in (torch.float32, torch.bfloat16) or not 8 <= c <= 2048 or c & (c - 1) or x.numel() <= c:
        return False
    if residual is not None and (not ordinary(residual) or residual.dtype != x.dtype or residual.shape != x.shape or residual.device != x.device
                                 or not _channels_last(residual)):
        return False
    return _channels_last(x)


def batch_norm_act(bn: nn.Module, x: torch.Tensor, residual: torch.Tensor | None = None,
                   relu: nn.Module | None = None, twice: bool = False):
    """``relu(bn(x) + residual)``; ``residual`` and ``relu`` may be left out.  With ``twice`` the result
    comes as a pair, for a caller that uses it in two places: the two gradients are then added inside
    the backward.  Fused for an
    ``nn.BatchNorm2d`` in training mode and a channels-last fp32 or bf16 ``x`` on the GPU with a
    power of two from 8 to 2048 channels; otherwise, and when one of the modules carries hooks or
    has been replaced, the modules are called."""
    if _fusable(bn, x, residual) and (relu is None or plain_module(relu, nn.ReLU)):
        return _BatchNormActFn.apply(x, residual, bn.weight, bn.bias, bn.running_mean, bn.running_var,
                                     bn.num_batches_tracked, bn.momentum, bn.eps, relu is not None, twice)
    y = bn(x)
    if residual is not None:
        y = y + residual
    y = y if relu is None else relu(y)
    return (y, y) if twice else y
