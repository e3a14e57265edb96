"""Max pooling of channels-last activations (``csrc/kernels/maxpool.cu``): one byte
per output element remembers which element of the window it was."""

from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _C
from ._plain import native, plain_module


class _MaxPoolFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, window, stride, pad):
        y, chosen = _C.max_pool_fwd(x, window, stride, pad)
        ctx.save_for_backward(x, chosen)
        ctx.geometry = (window, stride, pad)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, chosen = ctx.saved_tensors
        if torch.is_grad_enabled():  # the graph of this backward is wanted: torch's own op has one
            with torch.enable_grad():
                return torch.autograd.grad(F.max_pool2d(x, *ctx.geometry), x, dy, create_graph=True)[0], None, None, None
        # Saved-tensor hooks may have brought x back in another layout (save_on_cpu with pinned memory).
        x, dy = (t.contiguous(memory_format=torch.channels_last) for t in (x, dy))
        return _C.max_pool_bwd(dy, x, chosen, *ctx.geometry), None, None, None


def _square(v) -> int | None:
    if isinstance(v, int):
        return v
    return v[0] if isinstance(v, tuple) and len(v) == 2 and v[0] == v[1] else None


def max_pool(pool: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """``pool(x)``; for an ``nn.MaxPool2d`` with a square window and a channels-last fp32 or bf16 ``x``
    on the GPU that wants a gradient, by the kernels of this package."""
    if (native(x) and plain_module(pool, nn.MaxPool2d) and x.dim() == 4 and x.requires_grad and torch.is_grad_enabled()
            and x.dtype in (torch.float32, torch.bfloat16) and x.shape[1] % 8 == 0 and 0 < x.numel() // 8 < 2 ** 31 - 1
            and x.is_contiguous(memory_format=torch.channels_last) and x.data_ptr() % 16 == 0
            and _square(pool.dilation) == 1 and not pool.ceil_mode and not pool.return_indices):
        window, stride, pad = _square(pool.kernel_size), _square(pool.stride), _square(pool.padding)
        if (None not in (window, stride, pad) and 1 <= window <= 16 and stride >= 1 and 0 <= 2 * pad <= window
                and min(x.shape[2:]) + 2 * pad >= window):
            return _MaxPoolFn.apply(x, window, stride, pad)
    return pool(x)
