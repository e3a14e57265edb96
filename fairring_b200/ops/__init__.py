"""Fused single-GPU ops used by the training drivers."""

from .optim import FlatAdamW  # noqa: F401
from .layernorm import FusedLayerNorm, add_layer_norm, add_layer_norm_pair, fused_layer_norm  # noqa: F401
from .batchnorm import batch_norm_act  # noqa: F401
from .embedding import tied_embedding  # noqa: F401
from .linear import linear, linear_gelu, vocab_logits  # noqa: F401
from .pool import max_pool  # noqa: F401
from .stem import stem_conv  # noqa: F401
from .cross_entropy import cross_entropy_keeping_logits, fused_cross_entropy  # noqa: F401
