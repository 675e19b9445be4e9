"""Native (block-tile) sparse attention module: the B200-first entry point.

Same call shape as the reference's sparse modules -- ``forward(query, key, value, mask, mat)``
-> ``(out, attn)`` with ``[B, H, L, d]`` tensors -- but without the reference's per-call costs:

* fp32 *or* bf16 elements (the reference forces fp32, models/attention.py:88-92);
* no transposed copies of K (forward) and V (backward) (models/attention_blockcuda.py:48,80);
* block CSR/CSC fixed once per layer (``set_mask``), not rebuilt per call (:26-43);
* P is kept as ``[BH, nnzb, bs, bs]`` tiles, which is what TMA and the tensor cores want;
* on the tensor-core engine, head-split *views* of the ``[B, L, H*d]`` projections (what
  ``split_heads`` returns, models/attention.py:131-139) are read in place and the output is written
  in the same form, so neither the head split nor ``combine_heads`` copies anything.

``attn`` is returned in that tile layout (use ``to_reference_order`` to compare with the
reference's element-CSR order).
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _lib, _ops
from ._lib import check, lib, ptr

_DTYPES = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}


class ProbsHandle:
    """What a fused forward that stores no probabilities hands back in place of them: the operands and the
    per-row log-sum-exp from which any part of P can be rebuilt (``mean_attention_map`` does, for the
    warm-up phase).  Valid until the module's next forward."""

    def __init__(self, q, k, lse, pen, heads):
        self.q, self.k, self.lse, self.pen, self.heads = q, k, lse, pen, heads


class BlockSparseAttention(nn.Module):
    def __init__(self, config, dtype=torch.float32, keypad: bool = False, engine: int = _lib.ENGINE_AUTO,
                 device=None, fused=None, return_probs: bool = True, recompute=None, block32: str = "auto"):
        super().__init__()
        if isinstance(recompute, str):                          # every word would count as True
            raise _lib.SpionError(f"recompute must be None, False or True, not {recompute!r}")
        self.d = config["head_dim"]
        self.H = config["num_head"]
        self.L = config["max_seq_len"]
        self.B = config["batch_size"]
        self.bs = config["block_size"]
        self.BH = self.B * self.H
        self.dtype = dtype
        self.keypad = keypad
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        kind = _lib.KIND_BLOCK_KPM if keypad else _lib.KIND_BLOCK
        h = lib.spion_create(kind, self.d, self.L, self.BH, self.bs, _DTYPES[dtype], self.device.index or 0)
        if not h:
            raise _lib.SpionError("spion_create failed (unsupported shape, or no CUDA device)")
        self.handle = _lib.c_void_p(h)
        # what the native host path knows of this module; it owns the handle (a backward can outlive the module)
        self._ctx = _ops.make_context(h, _ops.NATIVE, self.B, self.H, self.L, self.d, self.device.index or 0,
                                      dtype == torch.bfloat16, keypad)
        self._ctx.owned = True
        check(lib.spion_set_engine(self.handle, engine), "spion_set_engine")
        self.engine = engine
        # 32-wide masks, bf16, head_dim 64, calls without stored probabilities: kernels on the mask's own blocks
        # ("own"), on 64-wide super-blocks ("super"), or chosen per mask by how full the gathered operands are
        check(lib.spion_set_block32_path(self.handle, {"auto": 0, "own": 1, "super": 2}[block32]), "spion_set_block32_path")
        self._ctx.needs_scratch = self.needs_scratch = bool(lib.spion_needs_scratch(self.handle))
        # fused kernels (S, P, dP, dS stay on chip) where the tensor-core engine covers the shape
        can_fuse = bool(lib.spion_supports_fused(self.handle))
        if fused and not can_fuse:
            raise _lib.SpionError("fused kernels need the tcgen05 engine (bf16, block 64, head_dim 32/64)")
        self.fused = can_fuse if fused is None else bool(fused)
        # return_probs=False (fused kernels only): the forward writes O and the log-sum-exp, nothing of size
        # nnz, and ``forward`` returns a ProbsHandle instead of the [BH, nnzb, bs, bs] tiles
        self.return_probs = bool(return_probs) or not self.fused
        # recompute=True (fused kernels): the backward rebuilds P and dS on chip from the log-sum-exp and nothing
        # of size nnz exists in memory; False: the forward stores P, the backward reads it and writes dS
        # (spion_attn_backward_ex).  None: chosen per mask in set_mask.
        self._recompute_arg = recompute
        self.recompute = self.fused and (recompute is None or bool(recompute))
        self.last = None
        self.nnzb = -1
        self._mask_key = _ops.ops.MaskKey()

    # settings the native host path reads: kept in its context
    @property
    def fused(self):
        return self._ctx.fused

    @fused.setter
    def fused(self, v):
        self._ctx.fused = bool(v)

    @property
    def recompute(self):
        return self._ctx.recompute

    @recompute.setter
    def recompute(self, v):
        self._ctx.recompute = bool(v)

    @property
    def return_probs(self):
        return self._ctx.return_probs

    @return_probs.setter
    def return_probs(self, v):
        self._ctx.return_probs = bool(v)

    # ------------------------------------------------------------------ pattern
    def set_mask(self, mat: torch.Tensor) -> int:
        """Fix the layer's block mask ([nb, nb], non-zero = selected).  Called once per layer at the
        dense->sparse switch, where the reference calls reconstruct_for_blocksparse."""
        m8 = (mat != 0).to(torch.uint8).contiguous().to(self.device)
        self._ctx.set_pattern(m8, self.bs)
        self.nnzb = int(lib.spion_pattern_nnzb(self.handle))
        if self.fused and self._recompute_arg is None:
            self.recompute = self._recompute_pays()
            self._ctx.rounded = not self.recompute and self._rebuilt_pays()
        from .pattern import pattern_from_mask
        self._pattern = pattern_from_mask(m8, self.bs)          # block CSR for the helpers above
        self._mask_key.set(mat)
        return self.nnzb

    def _recompute_pays(self) -> bool:
        """Which gradients serve the current mask: those of P as the log-sum-exp gives it (True), or those of the P that is rounded to bf16
        (False), bit for bit what stored tiles give (see _rebuilt_pays).

        No P returned: the first, whose forward is faster (forward + backward on one B200, us, against the second from rebuilt tiles; head_dim
        64 and 64 matrices unless stated): L = 4096, 3 % (two blocks per row) 143, 148; 5 % 162, 189; 30 % 540, 761; L = 16384, 5 % 1440, 2185;
        512 matrices, L = 1024, two blocks per row 314, 331; 2 matrices, L = 4096, 5 % 23, 28.  head_dim 32: 9 matrices, L = 9472, 12 % 139, 199;
        28 matrices, L = 6528, 4 % 92, 122; 2 matrices, L = 2048 17, 18.

        P returned: the second.  The gradients are those of the very P that the caller holds, and a change of it before the backward is
        an error.  The first differ by 4e-3 in norm, since dS comes from P before it is rounded (error against fp64 2.4e-3 instead of
        3.1e-3): recompute=True asks for them.  32-wide blocks and the full mask are on the first in any case.

        head_dim 32 with fewer than 2^15 selected blocks in all matrices: the second, although the first is faster there too (the
        three cases above).  P is normalised before and not after it is rounded to bf16, and a training step of the encoder classifier at
        such sizes multiplies any change of rounding: the gradients of the eighth pass over one batch of 8 pairs moved by 2e-3 to
        3.3e-1 of their norm over eight seeds (both paths are equally far from the fp32 step).  The bound is a line between measured
        sizes that leaves those steps as they were; it is no property of the kernels, and recompute=True takes the faster path
        below it as well.  The rule is the same for attention layers and for direct calls: one problem, one result."""
        nb = self.L // self.bs
        if self.bs == 32 or self.nnzb == nb * nb:
            return True
        return not self.return_probs and (self.d == 64 or self.BH * self.nnzb >= 1 << 15)

    def _rebuilt_pays(self) -> bool:
        """The gradients of the rounded P come from tiles that the backward rebuilds from two factors per row (True), or from stored P and dS, in
        the same bits.  Rebuilding costs the penalties and the exponentials twice more, storing costs the traffic, so short rows, small calls and padded keys
        are for stored tiles.  Forward + backward, us, rebuilt and stored, head_dim 32 (64), 64-wide blocks:
        no padding: 254 blocks in two-block rows 18.0, 15.9 (19.1, 16.8); 496 20.5, 19.1 (22.1, 21.5); 992 24.9, 27.0 (29.3, 30.3); 616 in rows of
          4.8 27.8, 31.3 (30.0, 33.2); 26240 in rows of 6.4 239, 307 (311, 366)
        padded keys, no P returned: 248 in two-block rows 25.0, 18.8; 1640 in rows of 3.2 48.2, 44.3; 2464 in rows of 4.8 58.6, 50.7; 4096 in rows of 4
          74.0, 76.5; 13120 in rows of 6.4 168, 184; 15872 in two-block rows 251, 244
        padded keys, P returned: 1640 in rows of 6.4 48.9, 45.8 (52.7, 49.4); 7936 in two-block rows 141, 133 (188, 176); 13120 in rows of 3.2 207, 199
          (261, 249), of 6.4 182, 184 (218, 216); 4916 in rows of 19 92.4, 99.2 (104, 107); 26240 in rows of 6.4 338, 347 (410, 412)"""
        blocks = self.BH * self.nnzb
        if not self.keypad:
            return blocks >= 512
        if not self.return_probs:
            return blocks >= 4096
        mean = self.nnzb / (self.L // self.bs)
        return blocks >= 4096 and mean >= 10 or blocks >= 16384 and mean >= 5

    @property
    def nnz(self) -> int:
        return self.nnzb * self.bs * self.bs

    def mean_attention_map(self, P_tiles) -> torch.Tensor:
        """A = mean over (b,h) of the probabilities of the last forward as an [L, L] fp32 map (zero outside the
        mask): what the encoder hands to pattern discovery (models/model_transformer.py:137), without a dense
        [B, H, L, L] tensor.  ``P_tiles`` is what ``forward`` returned beside the output: the
        [BH, nnzb, bs, bs] tiles, or a ProbsHandle, in which case the map is rebuilt from Q, K and the
        log-sum-exp and no probability was ever stored."""
        if isinstance(P_tiles, ProbsHandle):
            h = P_tiles
            A = torch.empty(self.L, self.L, dtype=torch.float32, device=h.q.device)
            check(lib.spion_set_stream(self.handle, _lib.current_stream_ptr()))
            check(lib.spion_set_head_layout(self.handle, h.heads), "spion_set_head_layout")
            check(lib.spion_mean_map_recompute(self.handle, ptr(h.q), ptr(h.k), ptr(h.lse), ptr(h.pen), ptr(A)),
                  "spion_mean_map_recompute")
            return A
        pat = self._pattern
        A = torch.empty(self.L, self.L, dtype=torch.float32, device=P_tiles.device)
        check(lib.spion_mean_map_tiles(ptr(P_tiles), _DTYPES[self.dtype], ptr(pat.blk_row), ptr(pat.col_idx), self.bs,
                                       self.nnzb, self.BH, self.L, ptr(A), _lib.current_stream_ptr()),
              "spion_mean_map_tiles")
        return A

    def launch_count(self) -> int:
        return int(lib.spion_launch_count(self.handle))

    def check_device_status(self) -> None:
        check(lib.spion_check_device_status(self.handle), "device status")

    def to_reference_order(self, P_tiles: torch.Tensor, mat: torch.Tensor) -> torch.Tensor:
        """[BH, nnzb, bs, bs] tiles -> the reference's [BH, nnz] element-CSR order."""
        nb = self.L // self.bs
        m = (mat != 0).to("cpu")
        out = []
        t = P_tiles.reshape(self.BH, self.nnzb, self.bs, self.bs)
        blk = 0
        for r in range(nb):
            n = int(m[r].sum())
            rows = t[:, blk:blk + n]                       # [BH, n, bs, bs]
            out.append(rows.permute(0, 2, 1, 3).reshape(self.BH, -1))
            blk += n
        return torch.cat(out, dim=1)

    # ------------------------------------------------------------------ call
    def use_mask(self, mat) -> None:
        """Make ``mat`` the current mask unless it already is (None: keep the current one)."""
        if mat is not None and not self._mask_key.matches(mat):
            self.set_mask(mat)
        if self.nnzb < 0:
            raise _lib.SpionError("no block mask set (call set_mask or pass mat)")

    def operand_form(self, t) -> int:
        """0: contiguous [B, H, L, d]; H: the head-split view of a contiguous [B, L, H, d] tensor; -1: neither."""
        if t.is_contiguous():
            return 0
        if tuple(t.stride()) == (self.L * self.H * self.d, self.d, self.H * self.d, 1):
            return self.H
        return -1

    def empty_operand(self, heads: int, device):
        """Uninitialised [B, H, L, d] tensor in the given form (see operand_form)."""
        if heads:
            return torch.empty(self.B, self.L, self.H, self.d, dtype=self.dtype, device=device).transpose(1, 2)
        return torch.empty(self.B, self.H, self.L, self.d, dtype=self.dtype, device=device)

    def result(self, out, probs, lse, pen, q, k, heads):
        """What a forward returns beside its output: the tiles, or a handle from which they can be rebuilt."""
        if lse is not None:
            self.last = ProbsHandle(q, k, lse, pen, heads)
        if not self.return_probs:
            return out, self.last
        return out, probs

    def forward(self, query, key, value, mask=None, mat=None):
        # The kernels take sizes from the context, not from the tensors: the call refuses any other shape, device or key-padding
        # mask with a SpionError (a short last batch would otherwise read and write past the buffers).
        self.use_mask(mat)
        return self.result(*_ops.attention(self._ctx, query, key, value, mask if self.keypad else None))


class DenseViaBlocks(nn.Module):
    """Warm-up (dense) attention through the same block kernels with the full mask: the dense phase of
    the reference (models/attention_cuda.py) without fp32 up-casts, transposed copies or a
    [B, H, L, L] tensor in the reference's S^T layout.  ``forward(query, key, value, mask)`` ->
    ``(out, probs)``; ``mean_attention_map(probs)`` gives the [L, L] map for pattern discovery.  On the
    tensor-core engine ``probs`` is a ProbsHandle: no probability is written in the whole dense phase."""

    def __init__(self, config, dtype=torch.float32, keypad: bool = False, device=None, return_probs: bool = False):
        super().__init__()
        self.block = BlockSparseAttention(config, dtype=dtype, keypad=keypad, device=device, return_probs=return_probs)
        nb = config["max_seq_len"] // config["block_size"]
        self.block.set_mask(torch.ones(nb, nb, dtype=torch.uint8, device=self.block.device))

    def forward(self, query, key, value, mask=None):
        return self.block(query, key, value, mask)

    def mean_attention_map(self, P_tiles):
        return self.block.mean_attention_map(P_tiles)
