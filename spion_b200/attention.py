"""Multi-head attention module: the host-side mirror of the reference's ``models/attention.py``.

``Attention(config, inference=False)`` has the reference's parameters (``W_q``, ``W_k``, ``W_v``,
``ff``), ``forward(X, mask, mat=None)`` -> ``(out, attn)``, and ``reconstruct_for_blocksparse
(config)`` which switches the layer from the dense warm-up path to the sparse path
(models/attention.py:105-129).  The four ``_*_compile_module`` loaders bind the same symbol
names with the same ``argtypes`` as the reference's (models/attention.py:141-191), but load the
shims built next to ``libspion_b200.so`` instead of ``./models/*.so``.

Config keys read: head_dim, num_head, max_seq_len, batch_size, block_size, task, transformer_dim
(the reference's), plus optional ``native`` (bool: use the block-tile kernels) and ``dtype``
("fp32" | "bf16", native only).
"""
from __future__ import annotations

import ctypes
import os
from ctypes import c_int

import torch
import torch.nn as nn

from . import _lib, _ops
from .attention_blockcuda import CUDABlockAttention
from .attention_blockcuda_mask import CUDABlockMaskAttention
from .attention_cuda import CUDAAttention
from .attention_cuda_mask import CUDAMaskAttention
from .layernorm import BiasGradLinear
from .native import BlockSparseAttention, DenseViaBlocks

# tasks whose inputs carry padding and therefore use the key-padding variants (models/attention.py:11)
mask_task = ['lra-listops', 'lra-text', 'lra-news', 'lra-yelp', 'lra-text1', 'lra-news1', 'lra-yelp1',
             'lra-text2', 'lra-news2', 'lra-yelp2', 'lra-retrieval']

_P = ctypes.c_void_p
_PLAIN_LINEAR = (nn.Linear, BiasGradLinear)
_DROPIN_DENSE = (CUDAAttention, CUDAMaskAttention)
_DROPIN_SPARSE = (CUDABlockAttention, CUDABlockMaskAttention)
_NATIVE_DENSE, _NATIVE_SPARSE = (DenseViaBlocks,), (BlockSparseAttention,)


def untouched(m, types) -> bool:
    """``m`` is of one of the types and a call that passes its forward over is no different: no hooks, no forward of its own."""
    if type(m) not in types:
        return False
    d = m.__dict__
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d)


def no_global_hooks() -> bool:
    return not nn.modules.module._has_any_global_hook()


def _load_shim(name, n_init, n_fwd, n_bwd, trailing_int):
    path = os.path.join(_lib.LIB_DIR, name)
    if not os.path.exists(path):
        raise ImportError(f"{path} is missing: run python -m spion_b200.build (there is no fallback)")
    cpp = ctypes.CDLL(path)
    cpp.init.argtypes = [c_int] * n_init
    cpp.init.restype = _P
    cpp.attn_forward.argtypes = [_P] * n_fwd + ([c_int] if trailing_int else [])
    cpp.attn_backward.argtypes = [_P] * n_bwd + ([c_int] if trailing_int else [])
    cpp.destroy.argtypes = [_P]
    return cpp


class Attention(nn.Module):
    def __init__(self, config, inference=False):
        super().__init__()
        self.inference = inference
        self.dim = config["transformer_dim"]
        self.head_dim = config["head_dim"]
        self.num_head = config["num_head"]
        self.seq_len = config["max_seq_len"]
        self.block_size = config["block_size"]
        self.num_blocks = int(self.seq_len / self.block_size)
        self.native = bool(config.get("native", False))
        self.native_dtype = torch.bfloat16 if config.get("dtype", "fp32") == "bf16" else torch.float32
        self.with_keypad = config["task"] in mask_task

        # same parameters and forward arithmetic as nn.Linear (models/attention.py:55-57); on the native path the
        # bias gradient of the backward is summed by the library's column-sum kernel
        Linear = BiasGradLinear if config.get("native") and config.get("fused_bias_grad", True) else nn.Linear
        self.W_q = Linear(self.dim, self.num_head * self.head_dim)
        self.W_k = Linear(self.dim, self.num_head * self.head_dim)
        self.W_v = Linear(self.dim, self.num_head * self.head_dim)

        if not inference and self.native:
            self.attn = DenseViaBlocks(config, dtype=self.native_dtype, keypad=self.with_keypad)
        elif not inference:
            num_batches = config["num_head"] * config["batch_size"]
            if self.with_keypad:
                attn_cpp = Attention._cuda_mask_compile_module()
                Dense = CUDAMaskAttention
            else:
                attn_cpp = Attention._cuda_compile_module()
                Dense = CUDAAttention
            attn_handle = attn_cpp.init(config["head_dim"], config["max_seq_len"], num_batches)
            if not attn_handle:
                raise _lib.SpionError("init() of the dense attention library returned NULL")
            self.attn = Dense(config, attn_cpp, attn_handle)

        self.ff = Linear(self.num_head * self.head_dim, self.dim)
        if torch.cuda.is_available():
            _lib.check(_lib.lib.spion_linear_prepare(int(self.native_dtype == torch.float32)), "spion_linear_prepare")

    def _untouched_stages(self, mat):
        """Weights, biases and attention module of a layer whose projections and attention are what was made here: nothing replaced,
        no hook that a one-node layer would pass over.  Else None.  (Looked up without nn.Module's __getattr__: 3 instead of 12 us.)"""
        if not no_global_hooks():
            return None
        mods, W, b = self._modules, [], []
        for name in ("W_q", "W_k", "W_v", "ff"):
            m = mods.get(name)
            if not untouched(m, _PLAIN_LINEAR):
                return None
            p = m._parameters
            W.append(p.get("weight"))
            b.append(p.get("bias"))
            if W[-1] is None or b[-1] is None:
                return None
        if mat is None and self.native:
            block = self.attn.block if untouched(self.attn, _NATIVE_DENSE) else None
        else:
            block = mods.get("attn" if mat is None else "block_attn")
        types = _NATIVE_SPARSE if self.native else _DROPIN_DENSE if mat is None else _DROPIN_SPARSE
        return (W, b, block) if untouched(block, types) else None

    def _one_node(self, X, mask, mat):
        """The whole layer as one autograd node on the library's kernels: projections, attention and output projection back to
        back in the layouts the next kernel reads.  None when something about the call is not served (the stages then run
        one by one): a width that is not a multiple of 32, another autocast dtype, replaced or hooked projections."""
        if torch.is_autocast_enabled():
            if not self.native or self.native_dtype != torch.bfloat16 or torch.get_autocast_dtype("cuda") != torch.bfloat16:
                return None
            fp32 = False
        else:
            if self.native and self.native_dtype != torch.float32:
                return None
            fp32 = True
        # in the dense phase the key bias has no effect: its gradient is the rounding noise of the stages, which the node leaves as it is
        noise = mat is None and fp32
        stages = self._untouched_stages(mat)
        if stages is None:
            return None
        W, b, block = stages
        if self.native:
            block.use_mask(mat)
            ctx = block._ctx
        elif mat is None:
            ctx = block.attn_func.context()
        else:
            ctx = block.context(mat)
        if not _ops.ops.layer_supported(ctx, X, W, b, fp32):
            return None
        out, P, lse, pen, q, k, heads = _ops.ops.attention_layer(ctx, X, mask if self.with_keypad else None, W, b, fp32, noise)
        if self.native:
            return block.result(out, P, lse, pen, q, k, heads)
        if mat is None:
            return out, P.permute(0, 1, 3, 2)
        return out, (0 if self.with_keypad else P)

    def forward(self, X, mask, mat=None):
        layer = self._one_node(X, mask, mat)
        if layer is not None:
            return layer
        # native dense phase in fp32: the products whose rounding the key bias's gradient consists of stay the framework's
        as_before = mat is None and self.native and not torch.is_autocast_enabled()

        def linear(m, x):
            return m(x, framework=True) if as_before and type(m) is BiasGradLinear else m(x)

        Q = self.split_heads(linear(self.W_q, X))
        K = self.split_heads(linear(self.W_k, X))
        V = self.split_heads(linear(self.W_v, X))
        with torch.autocast(device_type="cuda", enabled=False):
            if mat is None and self.native:
                attn_out, attn = self.attn(Q, K, V, mask.float())
                attn_out = attn_out.to(X.dtype)
            elif mat is None:
                call = None
                if untouched(self.attn, _DROPIN_DENSE) and no_global_hooks():
                    call = _ops.ops.attention(self.attn.attn_func.context(), Q.float(), K.float(), V.float(), mask if self.with_keypad else None)
                if call is not None:
                    attn_out, attn = call[0], call[1].permute(0, 1, 3, 2)
                else:
                    attn_out, attn = self.attn(Q.float(), K.float(), V.float(), mask.float())
            elif self.native:
                attn_out, attn = self.block_attn(Q, K, V, mask.float(), mat)
                attn_out = attn_out.to(X.dtype)
            else:
                attn_out, attn = self.block_attn(Q.float(), K.float(), V.float(), mask.float(), mat)
        attn_out = self.combine_heads(attn_out)
        out = linear(self.ff, attn_out)
        return out, attn

    def reconstruct_for_blocksparse(self, config):
        num_batches = int(config["num_head"] * config["batch_size"])
        model_dev = next(self.parameters()).device
        if self.native:
            # the layer above ignores the probabilities of the sparse phase (models/model_transformer.py:137 reads
            # them in the dense phase only): none are stored
            self.block_attn = BlockSparseAttention(config, dtype=self.native_dtype, keypad=self.with_keypad,
                                                   device=model_dev, return_probs=False)
            return
        if self.with_keypad:
            block_attn_cpp = Attention._blockcuda_mask_compile_module()
            Sparse = CUDABlockMaskAttention
        else:
            block_attn_cpp = Attention._blockcuda_compile_module()
            Sparse = CUDABlockAttention
        with torch.cuda.device(model_dev):
            handle = block_attn_cpp.init(config["head_dim"], config["max_seq_len"], num_batches, config["block_size"])
        if not handle:
            raise _lib.SpionError("init() of the block attention library returned NULL (is max_seq_len a multiple "
                                  "of block_size?)")
        self.block_attn = Sparse(config, block_attn_cpp, handle)
        self.block_attn.to(model_dev)

    def combine_heads(self, X):
        X = X.transpose(1, 2)
        return X.reshape(X.size(0), X.size(1), self.num_head * self.head_dim)

    def split_heads(self, X):
        X = X.reshape(X.size(0), X.size(1), self.num_head, self.head_dim)
        return X.transpose(1, 2)

    # ---- loaders: same symbols and argtypes as models/attention.py:141-191 -------------------
    @staticmethod
    def _cuda_compile_module():
        return _load_shim("attn.so", 3, 6, 12, False)

    @staticmethod
    def _blockcuda_compile_module():
        return _load_shim("block_attn.so", 4, 9, 14, True)

    @staticmethod
    def _cuda_mask_compile_module():
        return _load_shim("attn_mask.so", 3, 7, 12, False)

    @staticmethod
    def _blockcuda_mask_compile_module():
        return _load_shim("block_attn_mask.so", 4, 10, 14, True)
