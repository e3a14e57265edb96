"""Token plus position embedding of a model whose token table is also its output
projection (``csrc/kernels/embedding.cu``).
"""

from __future__ import annotations

import torch
import torch.nn as nn

from .. import _C
from ._plain import FUSE_FROM, native, ordinary, plain_module


class _TiedEmbeddingFn(torch.autograd.Function):
    """The embedded tokens and the table's bf16 copy for the projection: one node for both uses of
    the table, so that its gradient is built once."""

    @staticmethod
    def forward(ctx, tokens, table, pos, rows):
        ctx.save_for_backward(tokens)
        ctx.set_materialize_grads(False)  # an unused output arrives as None, not as zeros
        ctx.vocab, ctx.positions, ctx.d = table.shape[0], pos.shape[0], table.shape[1]
        low = table.new_empty((rows, ctx.d), dtype=torch.bfloat16)
        low[: ctx.vocab].copy_(table)
        if rows > ctx.vocab:
            low[ctx.vocab:].zero_()
        return _C.embed_fwd(tokens, table, pos), low

    @staticmethod
    def backward(ctx, dx, dlow):
        (tokens,) = ctx.saved_tensors
        if dx is None and dlow is None:
            return None, None, None, None
        dlow = None if dlow is None else dlow[: ctx.vocab]
        if torch.is_grad_enabled():  # the graph of this backward is wanted: torch's own ops have one
            scatter = torch.ops.aten.embedding_dense_backward
            dtable = dlow.float() if dlow is not None else None
            if dx is None:
                return None, dtable, None, None
            rows = scatter(dx, tokens, ctx.vocab, -1, False)
            places = torch.arange(tokens.shape[1], device=tokens.device).expand_as(tokens)
            dpos = scatter(dx, places, ctx.positions, -1, False)
            return None, rows if dtable is None else dtable + rows, dpos, None
        dx = None if dx is None else dx.contiguous()
        dlow = None if dlow is None else dlow.contiguous()
        dtable, dpos = _C.embed_bwd(dx, dlow, tokens, ctx.vocab, ctx.positions, ctx.d)
        return None, dtable, dpos, None


def _plain_table(m: nn.Module) -> bool:
    return (plain_module(m, nn.Embedding) and ordinary(m.weight) and m.padding_idx is None and m.max_norm is None and not m.sparse
            and not m.scale_grad_by_freq and m.weight.requires_grad and m.weight.dtype == torch.float32
            and m.weight.is_contiguous() and m.weight.data_ptr() % 16 == 0)


# Table elements from which rows are padded: below, the head's products are bound by their launches.
_PAD_FROM = FUSE_FROM


def tied_embedding(tok: nn.Embedding, pos: nn.Embedding, tokens: torch.Tensor, pad_rows: bool = False):
    """``(tok(tokens) + pos(0, 1, ...), table)``: ``table`` is what the output projection multiplies
    with, ``tok.weight`` or, where the fused form applies, its bf16 copy, with ``pad_rows`` and a large table
    with rows of zeros behind it up to a multiple of 8 (see :func:`fairring_b200.ops.vocab_logits`).  Fused in training under bf16
    autocast on the GPU.  The gradients of equal tokens are added in an order that the tokens fix: a step
    repeats itself bit for bit."""
    if (native(tokens) and tokens.dim() == 2 and tokens.dtype == torch.long and tokens.numel() > 0
            and torch.is_grad_enabled() and torch.is_autocast_enabled("cuda")
            and torch.get_autocast_dtype("cuda") == torch.bfloat16 and _plain_table(tok) and _plain_table(pos)
            and tok.weight.device == pos.weight.device == tokens.device and tok.embedding_dim == pos.embedding_dim
            and tok.embedding_dim % 8 == 0 and tokens.shape[1] <= pos.num_embeddings):
        rows = tok.num_embeddings
        rows = (rows + 7) // 8 * 8 if pad_rows and tok.weight.numel() >= _PAD_FROM else rows
        return _TiedEmbeddingFn.apply(tokens.contiguous(), tok.weight, pos.weight, rows)
    return tok(tokens) + pos(torch.arange(tokens.shape[1], device=tokens.device)), tok.weight
