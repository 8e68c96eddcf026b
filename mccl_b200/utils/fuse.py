"""When a fused node may stand for a module: only where nothing a user has put in its place would be passed by."""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

try:
    from torch.nn.modules.module import _has_any_global_hook
except ImportError:                       # not a public name: without it, nothing is fused
    def _has_any_global_hook() -> bool:
        return True

try:                                      # `with torch.device(...)` and torch.set_default_device: a mode that only places new tensors
    from torch.overrides import _get_current_function_mode_stack as _modes
    from torch.utils._device import DeviceContext as _DeviceContext
except ImportError:
    _modes = None
_mode_count = getattr(torch._C, "_len_torch_function_stack", lambda: 1)

_FUNCTIONS = ("linear", "embedding", "layer_norm", "gelu", "silu", "softmax", "scaled_dot_product_attention", "cross_entropy")
_STOCK = tuple(getattr(F, n) for n in _FUNCTIONS)
_PLAIN = (torch.Tensor, nn.Parameter)     # others may have a __torch_function__ of their own


def undisturbed() -> bool:
    """Whether the functions a module would call are torch's own and nobody watches their calls: no compiler, autocast, hooks for every
    module, or __torch_function__ mode."""
    if torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or _has_any_global_hook():
        return False
    if _mode_count() and (_modes is None or any(type(m) is not _DeviceContext for m in _modes())):
        return False
    return (F.linear, F.embedding, F.layer_norm, F.gelu, F.silu, F.softmax, F.scaled_dot_product_attention, F.cross_entropy) == _STOCK


def may_fuse(x: torch.Tensor, *others: torch.Tensor) -> bool:
    """Whether the kernels' nodes may take x, with these others, here."""
    return x.is_cuda and type(x) in _PLAIN and all(type(t) in _PLAIN for t in others) and undisturbed()


def as_made(m: nn.Module, cls: type) -> bool:
    """Whether calling m runs `cls.forward` and nothing else: not a subclass (a wrapper, a parametrised layer), no forward of
    its own, no hooks, no weights of a class of their own, and none of an embedding's options."""
    d = m.__dict__
    if type(m) is not cls or "forward" in d or d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]:
        return False
    for p in d["_parameters"].values():
        if p is not None and type(p) not in _PLAIN:
            return False
    return cls is not nn.Embedding or (m.padding_idx is None and m.max_norm is None and not m.scale_grad_by_freq and not m.sparse)
