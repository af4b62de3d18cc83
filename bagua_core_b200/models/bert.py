"""BERT-large encoder with a span-prediction (SQuAD-style) head: 24 layers, hidden 1024,
16 heads, FFN 4096, vocabulary 30522, post-LayerNorm, learned positions.  Attention goes
through `torch.nn.functional.scaled_dot_product_attention` (library kernel).  Random
initialisation only.

The encoder's projections are `ShadowLinear` modules: `nn.Linear` (same parameter names, same
math) unless an optimizer keeps bf16 copies of the weights (`FlatSGD(bf16_shadow=True)`) or
in-place weight-gradient accumulation is on (`bagua_core_b200.ops.wgrad.enabled`), in which case
they skip the per-forward weight casts and the cast-and-add of every weight gradient.

Under bf16 autocast on a GPU what lies between the projections runs as this package's kernels
(`csrc/kernels/encoder_ops.h`) and the library's LayerNorm in native autograd functions: the embedding
sum and the gradients of its tables, GELU with the projection in front of it, the packing of the attention
gradients, the span loss.  The roundings are those of the plain composition below, which runs elsewhere."""
from __future__ import annotations

from dataclasses import dataclass

import torch
import torch.nn as nn
import torch.nn.functional as F

from .._native import C as _C
from ..ops import wgrad
from ..ops.fused_linear import ShadowLinear
from ..ops.modules import drops_nothing, plain_embedding, untouched


_EMBED_TOKENS = _C.max_embedding_tokens  # more tokens per batch take the framework's embedding


@dataclass
class BertConfig:
    vocab_size: int = 30522
    hidden: int = 1024
    layers: int = 24
    heads: int = 16
    ffn: int = 4096
    max_pos: int = 512
    type_vocab: int = 2
    dropout: float = 0.1
    eps: float = 1e-12
    # True: LayerNorm as autocast runs it, fp32 in and out, which turns the whole residual stream
    # into fp32 and adds a cast before every projection.
    fp32_layernorm_io: bool = False

    @staticmethod
    def large():
        return BertConfig()

    @staticmethod
    def tiny():
        return BertConfig(vocab_size=1000, hidden=64, layers=2, heads=4, ffn=128, max_pos=128)


class _LayerNorm(nn.LayerNorm):
    """LayerNorm whose output stays in the autocast dtype.

    Autocast runs `layer_norm` in fp32: a bf16 activation is cast up, normalised, and leaves as
    fp32, so the residual sum that follows is fp32 too and every projection casts its input down
    again: per site about five times the bytes of a bf16-in, bf16-out normalisation.  The library
    kernel accumulates its statistics in fp32 whatever the input type, so here a low-precision
    input is normalised as it is (parameters cast to its type: 2·hidden values) and an fp32 input
    (the embedding sum) is normalised in fp32 and cast once.  Outside autocast this is
    `nn.LayerNorm`."""

    def forward(self, x):
        dev = x.device.type
        if not torch.is_autocast_enabled(dev):
            return super().forward(x)
        dtype = torch.get_autocast_dtype(dev)
        with torch.autocast(dev, enabled=False):
            if x.dtype == torch.float32:
                return F.layer_norm(x, self.normalized_shape, self.weight, self.bias, self.eps).to(dtype)
            return F.layer_norm(x, self.normalized_shape, self.weight.to(x.dtype), self.bias.to(x.dtype), self.eps)


def _bf16_autocast(x: torch.Tensor) -> bool:
    return x.is_cuda and torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16


def _fused(x: torch.Tensor, ln: nn.LayerNorm) -> bool:
    """Whether the fused kernels take this activation and the normalisation: bf16 autocast on a GPU, fp32 parameters."""
    return (_bf16_autocast(x) and untouched(ln, _LayerNorm) and ln.weight.dtype == torch.float32
            and ln.weight.shape[0] % 8 == 0)  # the kernels move 8 bf16 values at a time, and rows of any length


def _layer_norm(c: "BertConfig") -> nn.LayerNorm:
    return (nn.LayerNorm if c.fp32_layernorm_io else _LayerNorm)(c.hidden, eps=c.eps)


class _Layer(nn.Module):
    def __init__(self, c: BertConfig):
        super().__init__()
        self.heads = c.heads
        self.qkv = ShadowLinear(c.hidden, 3 * c.hidden)
        self.proj = ShadowLinear(c.hidden, c.hidden)
        self.ln1 = _layer_norm(c)
        self.fc1 = ShadowLinear(c.hidden, c.ffn)
        self.fc2 = ShadowLinear(c.ffn, c.hidden)
        self.ln2 = _layer_norm(c)
        self.drop = nn.Dropout(c.dropout)
        self.p = c.dropout

    def forward(self, x):
        b, s, h = x.shape
        m = self._modules
        ln1, ln2 = m.get("ln1"), m.get("ln2")
        if (x.dtype == torch.bfloat16 and _fused(x, ln1) and untouched(ln2, _LayerNorm) and (h // self.heads) % 8 == 0
                and x.numel() > 0):
            keep = drops_nothing(m.get("drop"))
            a = self.proj(_C.attention(self.qkv(x), self.heads, self.p if self.training else 0.0))
            x = self._add_norm(ln1, x, a if keep else self.drop(a))
            fc1 = self.fc1
            f = self.fc2(fc1(x, "gelu") if untouched(fc1, ShadowLinear) else F.gelu(fc1(x)))
            return self._add_norm(ln2, x, f if keep else self.drop(f))
        q, k, v = self.qkv(x).view(b, s, 3, self.heads, h // self.heads).permute(2, 0, 3, 1, 4)
        a = F.scaled_dot_product_attention(q, k, v, dropout_p=self.p if self.training else 0.0)
        a = a.transpose(1, 2).reshape(b, s, h)
        x = self.ln1(x + self.drop(self.proj(a)))
        f = self.fc2(F.gelu(self.fc1(x)))
        return self.ln2(x + self.drop(f))

    @staticmethod
    def _add_norm(ln, x, branch):
        return _C.add_layer_norm(x, branch, ln.weight, ln.bias, ln.eps, wgrad.active())


class BertForQuestionAnswering(nn.Module):
    def __init__(self, config: BertConfig = None):
        super().__init__()
        c = config or BertConfig.large()
        self.config = c
        self.tok = nn.Embedding(c.vocab_size, c.hidden)
        self.pos = nn.Embedding(c.max_pos, c.hidden)
        self.typ = nn.Embedding(c.type_vocab, c.hidden)
        self.ln = _layer_norm(c)
        self.drop = nn.Dropout(c.dropout)
        self.layers = nn.ModuleList([_Layer(c) for _ in range(c.layers)])
        self.qa = nn.Linear(c.hidden, 2)
        self.apply(self._init)

    @staticmethod
    def _init(m):
        if isinstance(m, (nn.Linear, nn.Embedding)):
            nn.init.normal_(m.weight, 0.0, 0.02)
            if isinstance(m, nn.Linear) and m.bias is not None:
                nn.init.zeros_(m.bias)

    def forward(self, input_ids, start_positions=None, end_positions=None):
        b, s = input_ids.shape
        m = self._modules
        if (plain_embedding(m.get("tok")) and plain_embedding(m.get("pos")) and _fused(self.tok.weight, m.get("ln"))
                and input_ids.is_cuda and input_ids.dtype == torch.int64 and 0 < b * s <= _EMBED_TOKENS and s <= self.pos.num_embeddings):
            x = _C.embed_layer_norm(input_ids, self.tok.weight, self.pos.weight, self.typ.weight, self.ln.weight,
                                    self.ln.bias, self.ln.eps, wgrad.active())
        else:
            pos = torch.arange(s, device=input_ids.device)
            x = self.ln(self.tok(input_ids) + self.pos(pos)[None] + self.typ.weight[0][None, None])
        x = self.drop(x)
        for layer in self.layers:
            x = layer(x)
        if (start_positions is not None and x.dtype == torch.bfloat16 and x.numel() > 0 and _bf16_autocast(x)
                and untouched(m.get("qa"), nn.Linear) and self.qa.out_features == 2
                and all(t.is_cuda and t.dtype == torch.int64 and t.dim() == 1 for t in (start_positions, end_positions))):
            logits = _C.linear(x, self.qa.weight, self.qa.bias, None, False)
            return _C.span_loss(logits, start_positions, end_positions)
        logits = self.qa(x).float()
        start, end = logits[..., 0], logits[..., 1]
        if start_positions is None:
            return start, end
        return (F.cross_entropy(start, start_positions) + F.cross_entropy(end, end_positions)) / 2
