"""When a fused node may stand for a module: only where nothing a user has put in its place would be passed by."""
from __future__ import annotations

import torch
from torch.nn.modules.module import _has_any_global_hook


def may_fuse(x: torch.Tensor) -> bool:
    """Whether the kernels' nodes may take x here: not while a compiler or autocast decides on the operations, and not past
    hooks that are called for every module."""
    return x.is_cuda and not torch.is_autocast_enabled("cuda") and not torch.compiler.is_compiling() and not _has_any_global_hook()


def as_made(m: torch.nn.Module, cls: type) -> bool:
    """Whether calling m runs `cls.forward` and nothing else: not a subclass (a wrapper, a parametrised layer), no forward of
    its own, no hooks."""
    d = m.__dict__
    return type(m) is cls and "forward" not in d and not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"]
                                                          or d["_backward_pre_hooks"])
