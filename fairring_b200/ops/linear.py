"""What surrounds the GEMMs of bf16 linear layers (``csrc/kernels/gelu.cu``): the
bias gradient as one pass over the gradient of the layer's output, and GELU,
whose backward adds the bias gradient up while it writes its result.

The products themselves are ``torch.nn.functional.linear``; only the bias is
taken out of its backward.
"""

from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _C
from ._plain import FUSE_FROM, native, ordinary, plain_module


class _LowWeightFn(torch.autograd.Function):
    """The weight's bf16 copy, which autocast would make as well; its gradient is widened by this
    package's kernel (19 us for 12.6 M elements, torch's cast takes 32 us)."""

    @staticmethod
    def forward(ctx, weight):
        return weight.to(torch.bfloat16)

    @staticmethod
    def backward(ctx, g):
        if torch.is_grad_enabled() or not g.is_contiguous() or g.data_ptr() % 16:
            return g.float()
        out = torch.empty_like(g, dtype=torch.float32)
        _C.bf16_grad_to_f32_(out, g)
        return out


def _product(fc: nn.Linear, x: torch.Tensor) -> torch.Tensor:
    weight = fc.weight
    if weight.dtype == torch.float32 and weight.requires_grad:
        weight = _LowWeightFn.apply(weight)
    return F.linear(x, weight, fc.bias.detach())


class _BiasGradFn(torch.autograd.Function):
    """The layer's output as it is; its backward gives the bias its gradient."""

    @staticmethod
    def forward(ctx, h, bias):
        ctx.bias_dtype = bias.dtype
        return h

    @staticmethod
    def backward(ctx, dh):
        if torch.is_grad_enabled():  # the graph of this backward is wanted: torch's own ops have one
            return dh, dh.flatten(0, -2).sum(0).to(ctx.bias_dtype)
        return dh, _C.column_sum(dh.contiguous(), ctx.bias_dtype)


class _GeluFn(torch.autograd.Function):
    """GELU of a layer's output, and the layer's bias gradient."""

    @staticmethod
    def forward(ctx, h, bias, tanh_form):
        ctx.tanh_form, ctx.bias_dtype = tanh_form, bias.dtype
        ctx.save_for_backward(h)
        return _C.gelu_fwd(h, tanh_form)

    @staticmethod
    def backward(ctx, dy):
        (h,) = ctx.saved_tensors
        if torch.is_grad_enabled():
            dh = torch.ops.aten.gelu_backward(dy, h, approximate="tanh" if ctx.tanh_form else "none")
            return dh, dh.flatten(0, -2).sum(0).to(ctx.bias_dtype), None
        dh, db = _C.gelu_bwd(dy.contiguous(), h, ctx.tanh_form, ctx.bias_dtype)
        return dh, db, None


# Output elements from which the fused forms are used: a two-layer model of width 128 (0.1 M elements) takes
# 2465 us a step without and 2640 us with them, while at 6 M elements the sum alone is 28 us against 12 us.
_FUSE_FROM = FUSE_FROM


def _fusable(fc: nn.Linear, x: torch.Tensor) -> bool:
    """Whether the layer's output will be bf16 on the GPU and large, and its bias wants a gradient."""
    if not ordinary(x) or x.dim() < 2 or x.numel() // max(1, x.shape[-1]) * fc.out_features < _FUSE_FROM:
        return False
    if not (native(x) and plain_module(fc, nn.Linear) and ordinary(fc.weight) and fc.bias is not None
            and fc.bias.requires_grad and torch.is_grad_enabled() and fc.out_features % 8 == 0
            and fc.bias.dtype in (torch.float32, torch.bfloat16) and fc.bias.device == x.device):
        return False
    if torch.is_autocast_enabled("cuda"):
        bf16 = torch.get_autocast_dtype("cuda") == torch.bfloat16
        bf16 = bf16 and x.dtype in (torch.float32, torch.bfloat16) and fc.weight.dtype in (torch.float32, torch.bfloat16)
    else:
        bf16 = x.dtype == fc.weight.dtype == fc.bias.dtype == torch.bfloat16
    return bf16


def linear(fc: nn.Linear, x: torch.Tensor) -> torch.Tensor:
    """``fc(x)``, with the bias gradient summed by one kernel where the output is bf16."""
    if not _fusable(fc, x):
        return fc(x)
    return _BiasGradFn.apply(_product(fc, x), fc.bias)


def linear_gelu(fc: nn.Linear, x: torch.Tensor, approximate: str = "none") -> torch.Tensor:
    """``F.gelu(fc(x), approximate=approximate)``; where the output is bf16, GELU is one kernel
    each way and its backward also sums the bias gradient."""
    if approximate not in ("none", "tanh") or not _fusable(fc, x):
        return F.gelu(fc(x), approximate=approximate)
    return _GeluFn.apply(_product(fc, x), fc.bias, approximate == "tanh")


class _PaddedHeadFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, table, bias):
        ctx.vocab, ctx.bias_dtype = bias.shape[0], bias.dtype
        ctx.save_for_backward(h, table)
        wide = torch.full((table.shape[0],), float("-inf"), dtype=table.dtype, device=bias.device)
        wide[: ctx.vocab].copy_(bias)
        return torch.addmm(wide, h, table.t())

    @staticmethod
    def backward(ctx, dl):
        h, table = ctx.saved_tensors
        narrow = dl[:, : ctx.vocab]
        if torch.is_grad_enabled():  # the graph of this backward is wanted: torch's own ops have one
            return narrow @ table[: ctx.vocab], dl.t() @ h, narrow.sum(0).to(ctx.bias_dtype)
        db = _C.column_sum(dl.contiguous(), ctx.bias_dtype)[: ctx.vocab].clone()
        return narrow.contiguous() @ table[: ctx.vocab], dl.t() @ h, db


def vocab_logits(h: torch.Tensor, table: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """``F.linear(h, table, bias)`` for a head whose bf16 ``table`` may have rows of zeros behind the
    vocabulary, up to a multiple of 8: the logits in those columns are minus infinity, probability 0.

    Rows of an odd number of logits start off the 16-byte boundaries that the tensor-core GEMMs
    need; for 1229 x 50265 logits of width 2048 the product takes 2.40 ms without padding and 0.18 ms
    with it, the weight gradient 1.49 and 0.18 ms.  The gradient of ``h`` is left to the product
    without padding (1.68 ms): another one's sums move the gradients of all layers below by 4 %
    at random weights."""
    if table.shape[0] == bias.shape[0]:
        return F.linear(h, table, bias)
    return _PaddedHeadFn.apply(h.to(table.dtype), table, bias)
