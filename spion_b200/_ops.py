"""The modules' host path in native code (csrc/torch_ops.cpp, built by ``python -m spion_b200.build``): autograd nodes that
call the C ABI.  There is no fallback: a missing extension raises."""
from __future__ import annotations

import importlib.util
import os

from . import _lib

PATH = os.path.join(_lib.LIB_DIR, "_torch_ops.so")


def _load():
    if not os.path.exists(PATH):
        raise ImportError(f"{PATH} is missing: run python -m spion_b200.build (there is no fallback)")
    spec = importlib.util.spec_from_file_location("_torch_ops", PATH)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


ops = _load()
NATIVE, DROPIN_SPARSE, DROPIN_DENSE = 0, 1, 2


def make_context(handle: int, mode: int, B: int, H: int, L: int, d: int, device: int, bf16: bool = False,
                 keypad: bool = False):
    c = ops.Context()
    c.handle, c.mode, c.B, c.H, c.L, c.d, c.device, c.bf16, c.keypad = handle, mode, B, H, L, d, device, bf16, keypad
    return c
