"""LayerNorm with the library's fused forward / backward kernels (csrc/ops/layer_norm.cu) for bf16 rows of 256, 512 or
1024 elements on CUDA; anything else goes through torch.nn.functional.layer_norm."""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _ext


def launches() -> int:
    return _ext.load().launches("norm")


_WIDTHS = (256, 512, 1024)


def fused_supported(x: torch.Tensor, weight: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and x.shape[-1] in _WIDTHS
            and weight.is_contiguous() and weight.data_ptr() % 16 == 0)


class FusedLayerNorm(nn.Module):
    """Drop-in for nn.LayerNorm over the last dimension (same parameter names)."""

    def __init__(self, d: int, eps: float = 1e-5):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(d))
        self.bias = nn.Parameter(torch.zeros(d))
        self.eps = eps

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        w, b = self.weight, self.bias
        if x.is_cuda and x.shape[-1] in _WIDTHS:
            y = _ext.load().layer_norm(x, w, b, self.eps)       # None where the kernels do not cover the case
            if y is not None:
                return y
        return F.layer_norm(x, x.shape[-1:], w, b, self.eps)
