"""Loader of the torch binding (csrc/torch): the C++ host side of the calls on torch tensors.

It is built next to libmccl.so by `python -m mccl_b200._build`, like the library itself, and links against it and torch.
"""
from __future__ import annotations

import importlib.machinery
import importlib.util
from pathlib import Path

import torch  # noqa: F401  (its libraries must be in the process before the binding is)

from . import _lib

_PATH = Path(__file__).resolve().parent / "lib" / "mccl_torch.so"
_mod = None


def load():
    """The binding, built in-tree first if it is not there yet."""
    global _mod
    if _mod is None:
        _lib.load()
        if not _PATH.exists():
            from . import _build
            _build.build()
        spec = importlib.util.spec_from_file_location("mccl_torch", _PATH, loader=importlib.machinery.ExtensionFileLoader("mccl_torch", str(_PATH)))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        _mod = mod
    return _mod
