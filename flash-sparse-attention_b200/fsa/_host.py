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
