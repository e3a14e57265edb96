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
    """False inside the transforms that look through torch's own ops but not through an
    ``autograd.Function`` around a native kernel: functorch (``vmap``, ``grad``, ``jvp``),
    forward-mode differentiation, tracing and compilation; and in inference mode."""
    return not (torch.is_inference_mode_enabled() or torch._C._are_functorch_transforms_active()
                or forward_ad._current_level >= 0 or torch.compiler.is_compiling() or torch.jit.is_tracing())


def plain_module(m: nn.Module, cls: type) -> bool:
    """Whether skipping ``m.__call__`` goes unnoticed: ``m`` is exactly a ``cls`` and nobody hooked it."""
    return (type(m) is cls and "forward" not in m.__dict__
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                     or _module._has_any_global_hook()))
