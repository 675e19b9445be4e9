"""The modules' host path in native code (csrc/torch_ops.cpp, built by ``python -m spion_b200.build``): autograd nodes that
call the C ABI.  There is no fallback: a missing extension raises."""
from __future__ import annotations

import importlib.util
import os

import torch

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


class _AttentionFn(torch.autograd.Function):
    """The attention node as one Python autograd function: what tracers record, and what refuses forward-mode tangents and function
    transforms."""

    @staticmethod
    def forward(ctx, query, key, value, mask, context, rest):
        leaves = [t.detach().requires_grad_(n) for t, n in zip((query, key, value), ctx.needs_input_grad)]
        with torch.enable_grad():
            out, probs, *others = ops.attention(context, *leaves, mask, True)
        rest.extend(others)
        ctx.inner = (out, [t for t in leaves if t.requires_grad])
        probs = out.new_empty(0) if probs is None else probs
        ctx.mark_non_differentiable(probs)
        ctx.set_materialize_grads(False)
        return out.detach(), probs

    @staticmethod
    def backward(ctx, grad_output, grad_probs):
        out, leaves = ctx.inner
        if grad_output is None or not leaves:
            return (None,) * 6
        grads = iter(torch.autograd.grad(out, leaves, grad_output, retain_graph=True))
        return tuple(next(grads) if n else None for n in ctx.needs_input_grad[:3]) + (None,) * 3


def attention(context, query, key, value, mask):
    """-> out, probabilities (None when none were stored), lse, penalties, Q and K as used, heads of their layout"""
    r = ops.attention(context, query, key, value, mask)
    if r is None:
        rest = []
        out, probs = _AttentionFn.apply(query, key, value, mask, context, rest)
        r = (out, probs if probs.numel() else None, *rest)
    return r


def make_context(handle: int, mode: int, B: int, H: int, L: int, d: int, device: int, bf16: bool = False,
                 keypad: bool = False):
    c = ops.Context()
    c.handle, c.mode, c.B, c.H, c.L, c.d, c.device, c.bf16, c.keypad = handle, mode, B, H, L, d, device, bf16, keypad
    return c
