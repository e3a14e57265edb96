"""The first convolution of an image network, 7 x 7 with stride 2 over 3 channels, as a
4 x 4 convolution over 2 x 2 pixel blocks (``csrc/kernels/stem.cu``).
"""

from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _C
from ._plain import native, plain_module

# Output pixels from which the fold pays: below, the launches that fold the weight cost the host more
# than the 0.35 ms per million pixels that the convolution gains.
_FOLD_FROM = 1 << 18


def _folded_weight(weight: torch.Tensor) -> torch.Tensor:
    """[out, 3, 7, 7] to bf16 [out, 16, 4, 4], laid out as the folded image's channels are."""
    w = F.pad(weight, (1, 0, 1, 0)).reshape(-1, 3, 4, 2, 4, 2)  # out, channel, block row, row, block column, column
    w = w.permute(0, 3, 5, 1, 2, 4).reshape(-1, 12, 4, 4)
    return F.pad(w, (0, 0, 0, 0, 0, 4)).to(dtype=torch.bfloat16, memory_format=torch.channels_last)


class _StemConvFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, images, weight):
        ctx.save_for_backward(images, weight)
        return F.conv2d(_C.stem_fold(images), _folded_weight(weight))

    @staticmethod
    def backward(ctx, dy):
        images, weight = ctx.saved_tensors
        dw = torch.ops.aten.convolution_backward(dy, images.to(torch.bfloat16), weight.to(torch.bfloat16), None, [2, 2],
                                                 [3, 3], [1, 1], False, [0, 0], 1, [False, True, False])[1]
        return None, dw.to(weight.dtype)


def stem_conv(conv: nn.Module, images: torch.Tensor) -> torch.Tensor:
    """``conv(images)``; folded for a plain 7 x 7, stride 2, padding 3 convolution of channels-last images
    that want no gradient, in training under bf16 autocast on the GPU."""
    if (native(images) and images.dim() == 4 and images.shape[1] == 3 and not images.requires_grad
            and plain_module(conv, nn.Conv2d) and conv.in_channels == 3 and conv.kernel_size == (7, 7)
            and conv.stride == (2, 2) and conv.padding == (3, 3) and conv.dilation == (1, 1) and conv.groups == 1
            and conv.bias is None and conv.padding_mode == "zeros" and conv.out_channels % 8 == 0
            and images.dtype in (torch.float32, torch.bfloat16) and conv.weight.dtype == torch.float32
            and conv.weight.device == images.device and conv.weight.requires_grad and torch.is_grad_enabled()
            and images.is_contiguous(memory_format=torch.channels_last) and torch.is_autocast_enabled("cuda")
            and torch.get_autocast_dtype("cuda") == torch.bfloat16
            and images.numel() // 12 >= _FOLD_FROM and images.numel() < 2 ** 31):
        return _StemConvFn.apply(images, conv.weight)
    return conv(images)
