"""Loader of the torch binding (csrc/torch): the C++ host side of the calls on torch tensors.

It is built next to libmccl.so by `python -m mccl_b200._build`, like the library itself, for the torch that is installed, and links
against both.
"""
from __future__ import annotations

import importlib.machinery
import importlib.util

import torch  # noqa: F401  (its libraries must be in the process before the binding is)

from . import _build, _lib

_mod = None


def load():
    """The binding, built in-tree first if it is not there yet."""
    global _mod
    if _mod is None:
        _lib.load()
        path = _build.ext_path(torch.__version__)
        if not path.exists():
            if torch.version.cuda is None:
                raise ImportError("the torch binding needs a torch with CUDA")
            _build.build()
        spec = importlib.util.spec_from_file_location("mccl_torch", path, loader=importlib.machinery.ExtensionFileLoader("mccl_torch", str(path)))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        _mod = mod
    return _mod


def load_if_built():
    """The binding where it is there and loads, None where not: for callers that do without."""
    if _mod is None and not _build.ext_path(torch.__version__).exists():
        return None
    try:
        return load()
    except (ImportError, OSError):
        return None
