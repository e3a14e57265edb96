"""Whether a call may be handed to an autograd function of this package."""

from __future__ import annotations

import torch
import torch.nn as nn
from torch.autograd import forward_ad
from torch.nn.modules import module as _module


# Elements from which the Python nodes of this package are used.  Below, torch's kernels are bound by
# their launches just as the package's are, and a Python node costs the host more than it saves.
FUSE_FROM = 1 << 22


def plain_autograd() -> bool:
    """False inside what looks through torch's own ops but not through a native kernel: tracing and
    compilation, dispatch modes (``make_fx``, fake tensors, FLOP counting), functorch (``vmap``,
    ``grad``, ``jvp``), forward-mode differentiation; and in inference mode."""
    if torch.compiler.is_compiling():  # asked first: Dynamo refuses some of the questions below
        return False
    return not (torch.jit.is_tracing() or torch._C._len_torch_dispatch_stack() > 0
                or torch.is_inference_mode_enabled() or torch._C._are_functorch_transforms_active()
                or forward_ad._current_level >= 0)


def ordinary(x) -> bool:
    """Neither a tracer's stand-in nor a tensor subclass, which may have no memory of its own."""
    return type(x) in (torch.Tensor, nn.Parameter)


def native(x) -> bool:
    """Whether a kernel may be handed ``x``: an ordinary tensor on the GPU, where nothing is traced.  To be
    asked before any other property of ``x``, which a tracer's stand-in does not answer."""
    return ordinary(x) and plain_autograd() and x.is_cuda


def plain_module(m: nn.Module, cls: type) -> bool:
    """Whether skipping ``m.__call__`` goes unnoticed: ``m`` is exactly a ``cls`` and nobody hooked it."""
    return (type(m) is cls and "forward" not in m.__dict__
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                     or _module._has_any_global_hook()))
