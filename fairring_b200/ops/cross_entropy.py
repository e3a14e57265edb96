"""Softmax cross-entropy for language-model heads
(``csrc/kernels/cross_entropy.cu``): the forward reads the logits once and keeps
one float per row, the backward writes the gradient in the logits' own dtype.

With a vocabulary that is a multiple of 8 the gradient is written over the
logits: they must not be used after the loss (their memory becomes their
gradient) -- true for a language-model head, where the loss is their only
consumer.  With any other vocabulary the logits are left alone.
"""

from __future__ import annotations

import torch
import torch.nn.functional as F

from .. import _C
from ._plain import native, plain_autograd


class _FusedCrossEntropyFn(torch.autograd.Function):
    """Where torch looks into an autograd function or refuses it; otherwise the same node is native,
    ``_C.cross_entropy``."""

    @staticmethod
    def forward(ctx, logits, targets):
        losses, lse = _C.cross_entropy_fwd(logits, targets)
        mean, count = _C.cross_entropy_mean(losses, targets, 1.0)
        ctx.save_for_backward(logits, targets, lse, count)
        return mean

    @staticmethod
    def backward(ctx, g):
        logits, targets, lse, count = ctx.saved_tensors
        if torch.is_grad_enabled():  # the graph of this backward is wanted
            return _C.cross_entropy_bwd_graph(logits, targets, g, count), None
        grad = logits.detach()
        _C.cross_entropy_bwd_(grad, targets, lse, g.float().reshape(1), 1.0, count)
        return grad, None


def fused_cross_entropy(logits: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
    """Mean cross-entropy of ``logits`` [rows, vocab] (fp32 or bf16) against
    ``targets`` [rows] (-100 is ignored; so is every other negative entry when the vocabulary is a
    multiple of 8, while with any other one it is an error as in ``F.cross_entropy``).  Consumes the logits when the
    vocabulary is a multiple of 8: after backward their storage holds the gradient (unless the
    backward's own graph was asked for).
    Falls back to ``F.cross_entropy(logits.float(), targets)`` off the GPU and for
    what the kernels do not take."""
    ok = (logits.is_cuda and logits.dim() == 2 and logits.is_contiguous()
          and logits.dtype in (torch.float32, torch.bfloat16) and targets.dtype == torch.long)
    if ok and logits.shape[1] % 8 == 0:
        targets = targets.contiguous()
        return _C.cross_entropy(logits, targets) if plain_autograd() else _FusedCrossEntropyFn.apply(logits, targets)
    return cross_entropy_keeping_logits(logits, targets)


def cross_entropy_keeping_logits(logits: torch.Tensor, targets: torch.Tensor, classes: int | None = None) -> torch.Tensor:
    """``F.cross_entropy(logits.float(), targets)`` by the same kernels; the logits stay as they are whatever
    the vocabulary.  With ``classes`` the logits from there on are padding."""
    if (native(logits) and logits.dim() == 2 and logits.is_contiguous() and logits.shape[1] > 0
            and logits.dtype in (torch.float32, torch.bfloat16) and logits.data_ptr() % 16 == 0
            and targets.dtype == torch.long and targets.shape == logits.shape[:1]
            and targets.device == logits.device):
        return _C.cross_entropy(logits, targets.contiguous(), logits.shape[1] if classes is None else classes)
    logits = logits if classes is None else logits[:, :classes]
    return F.cross_entropy(logits.float(), targets, ignore_index=-100)
