"""RoBERTa-style bidirectional transformer encoder with a masked-LM head: the
1.3B workload (24 layers, d_model 2048, 32 heads, FFN 8192, vocab 50265, seq
512) used to exercise the backend with ranks grouped as 4 machines x 2 GPUs.
Post-LayerNorm blocks as in BERT/RoBERTa, learned positions, tied decoder.
"""

from __future__ import annotations

from dataclasses import dataclass

import torch
import torch.nn as nn
import torch.nn.functional as F

from ..ops import add_layer_norm_pair, cross_entropy_keeping_logits, linear, linear_gelu, tied_embedding, vocab_logits
from ..ops import _plain
from ..ops._plain import native, plain_module


@dataclass
class EncoderConfig:
    n_layer: int = 24
    d_model: int = 2048
    n_head: int = 32
    d_ff: int = 8192
    vocab: int = 50265
    seq_len: int = 512
    mask_prob: float = 0.15

    @staticmethod
    def roberta_1p3b() -> "EncoderConfig":
        return EncoderConfig()

    @staticmethod
    def tiny() -> "EncoderConfig":
        return EncoderConfig(n_layer=2, d_model=128, n_head=4, d_ff=512, vocab=1000, seq_len=32)


class EncoderLayer(nn.Module):
    def __init__(self, cfg: EncoderConfig):
        super().__init__()
        self.n_head = cfg.n_head
        self.qkv = nn.Linear(cfg.d_model, 3 * cfg.d_model)
        self.proj = nn.Linear(cfg.d_model, cfg.d_model)
        self.ln1 = nn.LayerNorm(cfg.d_model)
        self.fc1 = nn.Linear(cfg.d_model, cfg.d_ff)
        self.fc2 = nn.Linear(cfg.d_ff, cfg.d_model)
        self.ln2 = nn.LayerNorm(cfg.d_model)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        b, s, d = x.shape
        q, k, v = self.qkv(x).view(b, s, 3, self.n_head, d // self.n_head).unbind(2)
        a = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2))
        x = self.ln1(x + self.proj(a.transpose(1, 2).reshape(b, s, d)))
        return self.ln2(x + self.fc2(F.gelu(self.fc1(x))))

    def forward_pair(self, x: torch.Tensor, low: torch.Tensor):
        """The same layer on the stream and its copy in the autocast dtype, which the linear layers read:
        takes and returns both, so that each LayerNorm's backward takes both gradients at once."""
        b, s, d = x.shape
        q, k, v = linear(self.qkv, low).view(b, s, 3, self.n_head, d // self.n_head).unbind(2)
        a = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2))
        x, low = add_layer_norm_pair(self.ln1, x, linear(self.proj, a.transpose(1, 2).reshape(b, s, d)))
        return add_layer_norm_pair(self.ln2, x, linear(self.fc2, linear_gelu(self.fc1, low)))


class EncoderMLM(nn.Module):
    def __init__(self, cfg: EncoderConfig):
        super().__init__()
        self.cfg = cfg
        self.tok = nn.Embedding(cfg.vocab, cfg.d_model)
        self.pos = nn.Embedding(cfg.seq_len, cfg.d_model)
        self.ln_emb = nn.LayerNorm(cfg.d_model)
        self.layers = nn.ModuleList(EncoderLayer(cfg) for _ in range(cfg.n_layer))
        self.head_dense = nn.Linear(cfg.d_model, cfg.d_model)
        self.head_ln = nn.LayerNorm(cfg.d_model)
        self.head_bias = nn.Parameter(torch.zeros(cfg.vocab))
        for m in self.modules():
            if isinstance(m, (nn.Linear, nn.Embedding)):
                nn.init.normal_(m.weight, std=0.02)
            if isinstance(m, nn.Linear):
                nn.init.zeros_(m.bias)

    def num_parameters(self) -> int:
        return sum(p.numel() for p in self.parameters())

    def forward(self, tokens: torch.Tensor, labels: torch.Tensor | None = None):
        """``labels``: target ids at masked positions, -100 elsewhere."""
        if not torch.jit.is_scripting():
            if native(tokens):
                return self._forward_native(tokens, labels)
        b, s = tokens.shape
        x = self.ln_emb(self.tok(tokens) + self.pos(torch.arange(s, device=tokens.device)))
        for layer in self.layers:
            x = layer(x)
        if labels is None:
            h = self.head_ln(F.gelu(self.head_dense(x)))
            return F.linear(h, self.tok.weight, self.head_bias)
        # Only masked positions go through the vocabulary projection.
        sel = labels.reshape(-1) != -100
        h = x.reshape(b * s, -1)[sel]
        h = self.head_ln(F.gelu(self.head_dense(h)))
        logits = F.linear(h, self.tok.weight, self.head_bias)
        return F.cross_entropy(logits.float(), labels.reshape(-1)[sel])

    def _forward_native(self, tokens: torch.Tensor, labels: torch.Tensor | None):
        """The same on the ops of this package."""
        b, s = tokens.shape
        x, table = tied_embedding(self.tok, self.pos, tokens, pad_rows=labels is not None)
        x = self.ln_emb(x)
        low = x
        # By the widest activation: below it forward_pair() would fuse little or nothing and cost the host more.
        large = x.is_cuda and b * s * max(self.cfg.d_ff, 3 * self.cfg.d_model) >= _plain.FUSE_FROM
        for layer in self.layers:
            if large and plain_module(layer, EncoderLayer):
                x, low = layer.forward_pair(x, low)
            else:
                x = low = layer(x)
        if labels is None:
            h = self.head_ln(F.gelu(self.head_dense(x)))
            return F.linear(h, table, self.head_bias)
        sel = labels.reshape(-1) != -100
        h = low.reshape(b * s, -1)[sel]
        h = self.head_ln(linear_gelu(self.head_dense, h))
        logits = vocab_logits(h, table, self.head_bias)
        return cross_entropy_keeping_logits(logits, labels.reshape(-1)[sel], self.head_bias.shape[0])


def mask_tokens(tokens: torch.Tensor, cfg: EncoderConfig, generator: torch.Generator, mask_id: int = 0):
    """15% of the positions are replaced by the mask id; labels keep the originals there."""
    pick = torch.rand(tokens.shape, generator=generator) < cfg.mask_prob
    labels = torch.where(pick, tokens, torch.full_like(tokens, -100))
    return torch.where(pick, torch.full_like(tokens, mask_id), tokens), labels
