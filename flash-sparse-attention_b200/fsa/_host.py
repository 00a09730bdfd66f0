"""The native host code (csrc/host): workspaces, launches and autograd of the operators, as one extension module.

It is built beside libfsa_sm100.so and calls that library through its C ABI; there is no fallback."""
from __future__ import annotations

import importlib.util
import os
import sys

import torch  # noqa: F401  (loads the libraries that the extension links against)

from fsa import _lib

PATH = os.path.join(os.path.dirname(_lib.LIB_PATH), "_fsa_host.so")

_mod = None


def host():
    """Load the extension once.  Raises if it has not been built."""
    global _mod
    if _mod is None:
        _lib.lib()
        if not os.path.exists(PATH):
            raise RuntimeError(f"{PATH} not found: build it with `python flash-sparse-attention_b200/build.py` (there is no fallback implementation)")
        spec = importlib.util.spec_from_file_location("_fsa_host", PATH)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        sys.modules["_fsa_host"] = mod
        _mod = mod
    return _mod


def plain_linear(m: torch.nn.Module) -> bool:
    """Nothing but ``x W^T``: no subclass, bias or hook that a call of the module would run.  Modules made of such parts run as
    one native function on their weights, others as their parts."""
    return type(m) is torch.nn.Linear and m.bias is None and not hooked(m)


def plain_gate(m: torch.nn.Module) -> bool:
    return (type(m) is torch.nn.Sequential and len(m) == 2 and plain_linear(m[0]) and type(m[1]) is torch.nn.Sigmoid
            and not hooked(m) and not hooked(m[1]))


def hooked(m: torch.nn.Module):
    return m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
