"""GPT-2 style decoder used as the data-parallel workload (24 layers, d_model 1024, 16 heads, FFN 4096,
vocab 50257, sequence 1024 for the "medium" shape, ~355M parameters).

Attention goes through scaled_dot_product_attention, the linear layers through cuBLAS.  On CUDA in bf16 everything
between them runs in this library's kernels, two autograd nodes per block (csrc/torch/gpt2.cc): a block hands on its
residual stream and its MLP output un-added, because the norm behind them adds them anyway.  Elsewhere the model is
plain PyTorch.  What the library adds around it is the communication (gradient buckets in symmetric memory,
all-reduced by the library's own kernels while backward still runs) and the fused optimizer step.
The token embedding is padded to a multiple of 64 rows so the tied output projection is tensor-core
friendly; the padding rows never receive probability mass (their logits are cut before the loss).
"""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _ext
from ..ops.norm import FusedLayerNorm
from ..utils.fuse import as_made, may_fuse


@dataclass
class GPT2Config:
    n_layer: int = 24
    d_model: int = 1024
    n_head: int = 16
    d_ff: int = 4096
    vocab_size: int = 50257
    seq_len: int = 1024
    dropout: float = 0.0

    @property
    def padded_vocab(self) -> int:
        return (self.vocab_size + 63) // 64 * 64

    @staticmethod
    def medium() -> "GPT2Config":
        return GPT2Config()

    @staticmethod
    def tiny() -> "GPT2Config":
        return GPT2Config(n_layer=2, d_model=128, n_head=4, d_ff=512, vocab_size=1000, seq_len=64)


def _added(x: torch.Tensor, pending, pending_bias) -> torch.Tensor:
    """x + pending in plain PyTorch, where the fused node that would have added them cannot run; the bias that is already
    part of `pending` gets its gradient here (its value is added and subtracted)."""
    if pending is None:
        return x
    return x + pending if pending_bias is None else x + pending + (pending_bias - pending_bias.detach())


class Block(nn.Module):
    grad_sink = False      # set by a data-parallel wrapper: fused nodes add weight gradients to .grad (csrc/torch/gradsink.h)

    def __init__(self, cfg: GPT2Config, fused: bool = True):
        super().__init__()
        norm = FusedLayerNorm if fused else nn.LayerNorm
        self.n_head = cfg.n_head
        self.ln1 = norm(cfg.d_model)
        # Separate q / k / v projections: same parameters and math as one 3d-wide projection, but the
        # backward pass gets three gradient GEMMs that accumulate into dx instead of a concatenation of
        # dq, dk, dv into one packed tensor (a pure copy that cost 7 % of the step).
        self.split_qkv = fused
        if fused:
            self.q = nn.Linear(cfg.d_model, cfg.d_model)
            self.k = nn.Linear(cfg.d_model, cfg.d_model)
            self.v = nn.Linear(cfg.d_model, cfg.d_model)
        else:
            self.qkv = nn.Linear(cfg.d_model, 3 * cfg.d_model)
        self.proj = nn.Linear(cfg.d_model, cfg.d_model)
        self.ln2 = norm(cfg.d_model)
        self.fc = nn.Linear(cfg.d_model, cfg.d_ff)
        self.out = nn.Linear(cfg.d_ff, cfg.d_model)

    _PARTS = (("ln1", FusedLayerNorm), ("q", nn.Linear), ("k", nn.Linear), ("v", nn.Linear), ("proj", nn.Linear), ("ln2", FusedLayerNorm),
              ("fc", nn.Linear), ("out", nn.Linear))

    def _params(self):
        """Weights and biases in the order the fused nodes take them; None where a part is not what this class made it."""
        mods, out = self._modules, []
        for name, cls in self._PARTS:
            m = mods.get(name)
            if m is None or not as_made(m, cls):
                return None
            p = m._parameters
            if p["bias"] is None:
                return None
            out += (p["weight"], p["bias"])
        return out if self.ln1.eps == self.ln2.eps else None

    def fused(self, x: torch.Tensor, pending, pending_bias, shape, bias_here: bool):
        """The block on x + pending ([tokens, d_model]) as two tensors still to be added, or None where it has to run as plain
        PyTorch.  `bias_here`: whether the gradient of the last bias is taken here or by whoever adds the two."""
        params = self._params() if self.split_qkv and may_fuse(x) else None
        if params is None:
            return None
        b, s = shape
        return _ext.load().gpt2_block(x, pending, pending_bias, params, b, s, self.n_head, bias_here,
                                      self.ln1.eps, self.grad_sink)

    def forward(self, x: torch.Tensor, pending=None, pending_bias=None, shape=None):
        """x [batch, seq, d_model] -> the same.  With `shape` = (batch, seq), as GPT2 calls it: x and `pending` are
        [batch * seq, d_model], the input is their sum, and the result is a pair whose sum is the output."""
        if shape is not None:
            pair = self.fused(x, pending, pending_bias, shape, False)
            if pair is not None:
                return pair
            x = _added(x, pending, pending_bias)
            return self._plain(x.view(*shape, -1)).view(x.shape), None
        if self.split_qkv and x.is_cuda and x.dim() == 3 and x.is_contiguous():
            pair = self.fused(x.view(-1, x.shape[-1]), None, None, x.shape[:2], True)
            if pair is not None:
                return (pair[0] + pair[1]).view(x.shape)
        return self._plain(x)

    def _plain(self, x: torch.Tensor) -> torch.Tensor:
        b, s, d = x.shape
        h = self.ln1(x)
        if self.split_qkv:
            q, k, v = (p(h).view(b, s, self.n_head, d // self.n_head).transpose(1, 2) for p in (self.q, self.k, self.v))
        else:
            q, k, v = self.qkv(h).view(b, s, 3, self.n_head, d // self.n_head).permute(2, 0, 3, 1, 4)
        a = F.scaled_dot_product_attention(q, k, v, is_causal=True)
        x = x + self.proj(a.transpose(1, 2).reshape(b, s, d))
        x = x + self.out(F.gelu(self.fc(self.ln2(x)), approximate="tanh"))
        return x


class GPT2(nn.Module):
    """Decoder-only transformer with learned positions, pre-LayerNorm blocks and a tied output projection;
    forward(idx, targets) returns the mean cross-entropy, forward(idx) the logits."""

    grad_sink = False      # see Block

    def __init__(self, cfg: GPT2Config, fused_loss: bool = True):
        super().__init__()
        self.cfg = cfg
        self.fused_loss = fused_loss      # the library's cross-entropy and LayerNorm kernels (CUDA, bf16); False = stock PyTorch
        self.wte = nn.Embedding(cfg.padded_vocab, cfg.d_model)
        self.wpe = nn.Embedding(cfg.seq_len, cfg.d_model)
        self.blocks = nn.ModuleList(Block(cfg, fused_loss) for _ in range(cfg.n_layer))
        self.ln_f = (FusedLayerNorm if fused_loss else nn.LayerNorm)(cfg.d_model)
        self.apply(self._init)
        for blk in self.blocks:  # GPT-2's scaled init of the residual projections
            nn.init.normal_(blk.proj.weight, std=0.02 / math.sqrt(2 * cfg.n_layer))
            nn.init.normal_(blk.out.weight, std=0.02 / math.sqrt(2 * cfg.n_layer))

    @staticmethod
    def _init(m: nn.Module) -> None:
        if isinstance(m, (nn.Linear, nn.Embedding)):
            nn.init.normal_(m.weight, std=0.02)
            if isinstance(m, nn.Linear) and m.bias is not None:
                nn.init.zeros_(m.bias)

    def num_params(self) -> int:
        return sum(p.numel() for p in self.parameters())

    def forward(self, idx: torch.Tensor, targets: torch.Tensor | None = None):
        b, s = idx.shape
        w = self.wte.weight
        x = None
        if self.fused_loss and w.dtype == torch.bfloat16 and may_fuse(w, idx) and as_made(self.wte, nn.Embedding) and as_made(self.wpe, nn.Embedding):
            x = _ext.load().decoder_embed(idx, w, self.wpe.weight, self.grad_sink)      # None where the kernels do not cover the case
        if x is not None:
            pending = bias = None
            for blk in self.blocks:
                if not as_made(blk, Block):                  # its caller's hooks or wrapper see a block as it is called elsewhere
                    x = blk(_added(x, pending, bias).view(b, s, -1)).reshape(b * s, -1)
                    pending = bias = None                    # it has added everything
                    continue
                x, pending = blk(x, pending, bias, (b, s))
                # a block that ran as plain PyTorch has added everything and taken its bias gradient itself
                bias = blk.out.bias if pending is not None else None
            x = self._final_norm(x, pending, bias if pending is not None else None)
        else:
            pos = torch.arange(s, device=idx.device)
            x = self.wte(idx) + self.wpe(pos)
            for blk in self.blocks:
                x = blk(x)
            x = self.ln_f(x)
        if targets is not None and self.fused_loss and x.dtype == torch.bfloat16 and may_fuse(x, w, targets):
            loss = _ext.load().decoder_head_loss(x.view(b * s, -1), w, targets, self.cfg.vocab_size, False, self.grad_sink)
            if loss is not None:
                return loss
        logits = F.linear(x, w).view(b, s, -1)           # tied output projection, padded vocab
        if targets is None:
            return logits[..., : self.cfg.vocab_size]
        flat = logits.view(b * s, -1)
        if self.fused_loss and flat.is_cuda and flat.dtype == torch.bfloat16:
            from ..ops.loss import fused_cross_entropy
            return fused_cross_entropy(flat, targets.reshape(-1).contiguous(), self.cfg.vocab_size)
        return F.cross_entropy(flat[:, : self.cfg.vocab_size].float(), targets.reshape(-1))

    def _final_norm(self, x: torch.Tensor, pending, bias) -> torch.Tensor:
        n = self.ln_f
        if pending is None:
            return n(x)
        h = None
        if as_made(n, FusedLayerNorm):
            h = _ext.load().gpt2_final_norm(x, pending, bias, n.weight, n.bias, n.eps, self.grad_sink)
        return h if h is not None else n(_added(x, pending, bias))
