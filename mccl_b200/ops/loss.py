"""Fused softmax cross-entropy for bf16 logits (csrc/ops/cross_entropy.cu): one read of the logits in the
forward pass, the gradient written in bf16 over the logits in the backward pass, no fp32 copy of the
rows x vocab matrix."""
from __future__ import annotations

import torch

from .. import _ext


def launches() -> int:
    return _ext.load().launches("loss")


def fused_cross_entropy(logits: torch.Tensor, targets: torch.Tensor, vocab: int | None = None) -> torch.Tensor:
    """Mean cross-entropy of bf16 `logits` [rows, width] against int64 `targets` [rows]; columns at or beyond
    `vocab` (padding of the output projection) take no probability mass and get zero gradient."""
    if not logits.is_cuda:
        raise RuntimeError("fused_cross_entropy runs on CUDA (sm_100a) only")
    assert logits.dim() == 2 and logits.dtype == torch.bfloat16 and logits.stride(1) == 1
    assert targets.dtype == torch.int64 and targets.is_contiguous() and targets.numel() == logits.shape[0]
    loss = _ext.load().cross_entropy(logits, targets, vocab)
    if loss is None:
        raise ValueError("fused_cross_entropy: logits and targets do not fit together")
    return loss
