"""The attention and discovery kernels at the sizes where their loops and dispatch rules end: lines of every length, empty lines,
full masks, one more and one fewer than what fills the chip, several maps per call."""
import numpy as np
import pytest
import torch

from oracle import attention as oatt
from oracle import csr as ocsr
from oracle import pattern as opat
from spion_b200 import synthetic

pytestmark = pytest.mark.gpu
# fp32: the reference's parity bound, max-abs
FP32_TOL = 1e-4
# bf16: P, dS and the results are rounded to 2^-9 each, and an output is a sum of products of two of them: at most 3 * 2^-9 = 6e-3
# of the sum of magnitudes, which exceeds the largest output by a factor of about three in these inputs
BF16_REL = 2e-2


def cfg(B, H, L, d, bs):
    return {"head_dim": d, "num_head": H, "max_seq_len": L, "batch_size": B, "block_size": bs, "transformer_dim": H * d, "task": "t"}


def far(a, b, relative):
    a, b = a.detach().float().cpu(), b.detach().float().cpu()
    return float((a - b).abs().max() / (b.abs().max().clamp_min(1e-30) if relative else 1.0))


def lines_of_every_length(nb, zero=True):
    """Row r has r + 1 blocks, column c nb - c; with `zero` one row and one column without any."""
    mat = np.tril(np.ones((nb, nb), dtype=np.uint8))
    if zero:
        mat[nb // 2, :] = 0
        mat[:, nb // 3] = 0
    return mat


def run(mod, Q, K, V, dO, mat, kp):
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    out, _ = mod(q, k, v, None if kp is None else kp.cuda(), torch.as_tensor(mat).cuda())
    out.backward(dO.cuda())
    mod.check_device_status()
    return out, q.grad, k.grad, v.grad


def compare(got, Q, K, V, dO, mat, bs, kp, tol, relative):
    O, _, gQ, gK, gV = oatt.sparse_attention(Q.float(), K.float(), V.float(), mat, bs, kp, dO.float())
    for name, a, b in zip(("O", "dQ", "dK", "dV"), got, (O, gQ, gK, gV)):
        assert far(a, b, relative) <= tol, f"{name}: {far(a, b, relative):.3e}"


@pytest.mark.parametrize("d,bs", [(64, 64), (32, 64), (32, 32)])
@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("case", ["lines", "full", "growing"])
def test_streaming_forward_and_backward(d, bs, padded, case):
    """No stored P: rows and columns of 1 to 11 blocks, none at all, an odd last pair; the full mask; scores that outgrow the
    maximum a row started with.  bs 32: the super-block form, with quarters of a block switched off."""
    from spion_b200.native import BlockSparseAttention
    B, H, nb = 2, 3, 11 if bs == 64 else 22
    L = nb * bs
    Q, K, V, dO = (t.to(torch.bfloat16) for t in synthetic.qkv(3 + d, B, H, L, d))
    if case == "growing":
        K = (K.float() * torch.linspace(0.5, 12.0, L)[:, None]).to(torch.bfloat16)
    mat = np.ones((nb, nb), np.uint8) if case == "full" else lines_of_every_length(nb, case == "lines")
    kp = synthetic.key_padding(5, B, L) if padded else None
    mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.bfloat16, keypad=padded, recompute=True, return_probs=False)
    got = run(mod, Q, K, V, dO, mat, kp)
    compare(got, Q, K, V, dO, mat, bs, kp, BF16_REL, True)
    with torch.no_grad():                                    # and without a backward
        out, _ = mod(Q.cuda(), K.cuda(), V.cuda(), None if kp is None else kp.cuda(), torch.as_tensor(mat).cuda())
    assert torch.equal(out, got[0].detach())


@pytest.mark.parametrize("d,nb", [(64, 5), (32, 5), (32, 1)])
def test_streaming_kernels_with_many_units(d, nb):
    """More than 32 block rows per CTA, some without entries: the records of a CTA's pairs are made 32 lines and 16 pairs at a time."""
    from spion_b200.native import BlockSparseAttention
    B, H, L = (400, 3, 5 * 64) if nb > 1 else (1900, 3, 64)
    Q, K, V, dO = (t.to(torch.bfloat16) for t in synthetic.qkv(7 + d, B, H, L, d))
    mat = lines_of_every_length(nb, True) if nb > 1 else np.ones((1, 1), np.uint8)
    kp = synthetic.key_padding(4, B, L)
    mod = BlockSparseAttention(cfg(B, H, L, d, 64), dtype=torch.bfloat16, keypad=True, recompute=True, return_probs=False)
    compare(run(mod, Q, K, V, dO, mat, kp), Q, K, V, dO, mat, 64, kp, BF16_REL, True)


# (bs, d, B, H, blocks per side): few threads' worth of work (four rows per thread), more (eight; columns split over clusters), many
# (eight; one CTA per column group); groups of four matrices with one, two and three left over
@pytest.mark.parametrize("bs,d,B,H,nb", [(32, 32, 1, 1, 1), (32, 64, 1, 3, 7), (64, 32, 1, 1, 2), (64, 64, 2, 1, 9),
                                         (32, 32, 50, 3, 8), (32, 64, 42, 5, 7), (64, 32, 40, 1, 8), (64, 64, 7, 5, 9),
                                         (32, 32, 301, 3, 8), (64, 64, 119, 3, 5),
                                         (32, 64, 2, 1, 3), (64, 64, 1, 2, 3), (64, 32, 1, 1, 3)])   # nb 3: the full mask's kernels
def test_fp32_fused_kernels(bs, d, B, H, nb):
    from spion_b200.native import BlockSparseAttention
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(17 + nb, B, H, L, d)
    mat = np.ones((3, 3), np.uint8) if nb == 3 else lines_of_every_length(nb, nb > 4)
    kp = synthetic.key_padding(9, B, L) if nb % 2 else None
    mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.float32, keypad=kp is not None)
    compare(run(mod, Q, K, V, dO, mat, kp), Q, K, V, dO, mat, bs, kp, FP32_TOL, False)


# (bs, d, B, H, blocks per side): block rows around what fits the chip at once with four, two and one group of threads per row
# (148 SMs: up to 296, up to 592, more), rows of one block, rows shorter than the groups
@pytest.mark.parametrize("bs,d,B,H,nb", [(32, 32, 1, 1, 9), (32, 64, 37, 1, 8), (32, 32, 33, 1, 9), (32, 64, 74, 1, 8), (32, 32, 66, 1, 9),
                                         (64, 32, 37, 1, 8), (64, 64, 33, 1, 9), (32, 32, 200, 2, 1)])
@pytest.mark.parametrize("layout", ["tiles", "csr"])
def test_fp32_rows_shared_by_groups(bs, d, B, H, nb, layout):
    from spion_b200.attention import Attention
    from spion_b200.attention_blockcuda import CUDABlockAttention
    from spion_b200.native import BlockSparseAttention
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(23 + nb, B, H, L, d)
    mat = lines_of_every_length(nb, nb > 4)
    if layout == "tiles":
        mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.float32)
        got = run(mod, Q, K, V, dO, mat, None)
        compare(got, Q, K, V, dO, mat, bs, None, FP32_TOL, False)
        return
    cpp = Attention._blockcuda_compile_module()                  # element CSR, backward without O (two passes over a row)
    handle = cpp.init(d, L, B * H, bs)
    mod = CUDABlockAttention(cfg(B, H, L, d, bs), cpp, handle)
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    out, _ = mod(q, k, v, torch.ones(B, L).cuda(), torch.as_tensor(mat.astype(np.float32)).cuda())
    out.backward(dO.cuda())
    compare((out, q.grad, k.grad, v.grad), Q, K, V, dO, mat, bs, None, FP32_TOL, False)
    cpp.destroy(handle)


# (bs, d, B, blocks per side, blocks per row, groups of threads per row forward, backward): both sides of one, one and a half, three and
# four block rows per SM (148 SMs), rows of one and two blocks
@pytest.mark.parametrize("bs,d,B,nb,per,forward,backward",
                         [(32, 32, 37, 4, 2, 4, 4), (32, 32, 30, 5, 2, 2, 2), (32, 64, 111, 4, 3, 2, 2), (32, 64, 89, 5, 3, 2, 1),
                          (32, 32, 148, 4, 2, 2, 2), (32, 64, 119, 5, 2, 1, 1), (32, 32, 40, 4, 1, 1, 1), (64, 64, 37, 4, 2, 2, 2),
                          (64, 32, 37, 6, 3, 2, 2), (64, 64, 45, 5, 3, 1, 1), (64, 64, 30, 5, 2, 1, 1), (64, 64, 20, 5, 1, 1, 1)])
def test_fp32_groups_per_row(bs, d, B, nb, per, forward, backward):
    from torch.profiler import ProfilerActivity, profile

    from spion_b200.native import BlockSparseAttention
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(29 + nb, B, 1, L, d)
    mat = np.zeros((nb, nb), np.uint8)
    for x in range(per):
        mat[np.arange(nb), (np.arange(nb) + x) % nb] = 1
    mod = BlockSparseAttention(cfg(B, 1, L, d, bs), dtype=torch.float32)
    mod.set_mask(torch.as_tensor(mat).cuda())
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        got = run(mod, Q, K, V, dO, mat, None)
        torch.cuda.synchronize()
    compare(got, Q, K, V, dO, mat, bs, None, FP32_TOL, False)
    names = {e.name for e in p.events()}
    for kernel, groups in (("fused_fwd_kernel", forward), ("fused_bwd_row_delta_kernel", backward)):
        assert any(f"{kernel}<{bs}, {d}, 4, {groups}>" in n for n in names), names


def fp32_kernels(step):
    from torch.profiler import ProfilerActivity, profile
    step()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        step()
        torch.cuda.synchronize()
    return {e.name for e in prof.events() if "mma_" in e.name or "fused_" in e.name}


def fp32_call(layout, B, H, L, d, bs, mat, kp):
    """One call per layout: block tiles; element CSR with the reference's signature (a backward without O: two passes over a row); element CSR
    through the layers' host path (with O)."""
    from spion_b200 import _ops
    from spion_b200.attention import Attention
    from spion_b200.attention_blockcuda import CUDABlockAttention
    from spion_b200.native import BlockSparseAttention
    if layout == "tiles":
        mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.float32, keypad=kp is not None)
        return lambda q, k, v: mod(q, k, v, None if kp is None else kp.cuda(), torch.as_tensor(mat).cuda())[0], lambda: None
    cpp = Attention._blockcuda_compile_module()
    handle = cpp.init(d, L, B * H, bs)
    mod = CUDABlockAttention(cfg(B, H, L, d, bs), cpp, handle)
    ones, fmat = torch.ones(B, L).cuda(), torch.as_tensor(mat.astype(np.float32)).cuda()
    if layout == "csr":
        return lambda q, k, v: mod(q, k, v, ones, fmat)[0], lambda: cpp.destroy(handle)
    return lambda q, k, v: _ops.attention(mod.context(fmat), q, k, v, None)[0], lambda: cpp.destroy(handle)


# Calls on the fp32 tensor-core kernels: (bs, d, B, H, blocks per side, full columns), one and two 16-row tiles per warp, groups of matrices with some
# left over, rows and columns of every length and none, full columns, key padding
LINES = [(32, 32, 65, 1, 9), (32, 32, 151, 3, 8), (32, 64, 33, 3, 7), (64, 32, 41, 1, 8), (64, 64, 31, 1, 11), (64, 64, 61, 1, 5)]
# full columns shared by clusters, six of them more than a launch has clusters along the columns
SHARED = [(32, 32, 65, 1, 20), (32, 32, 151, 3, 16), (32, 64, 33, 3, 15), (64, 32, 41, 1, 17), (64, 64, 31, 1, 18)]


@pytest.mark.parametrize("bs,d,B,H,nb,full", [c + (n,) for c in LINES for n in (0, 2)] + [c + (n,) for c in SHARED for n in (2, 6)])
@pytest.mark.parametrize("layout", ["tiles", "csr", "csr with O"])
def test_fp32_tensor_core_kernels(bs, d, B, H, nb, full, layout):
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(37 + nb, B, H, L, d)
    mat = lines_of_every_length(nb) if not full else synthetic.band_random_mask(3, nb, 0.0)
    if full:
        mat[:, 1:full] = 1
        mat[:, nb - 1] = 1
    kp = synthetic.key_padding(9, B, L) if nb % 2 and layout == "tiles" else None
    call, close = fp32_call(layout, B, H, L, d, bs, mat, kp)
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    got = []

    def step():
        out = call(q, k, v)
        got[:] = (out,) + torch.autograd.grad(out, (q, k, v), dO.cuda())

    names = fp32_kernels(step)
    close()
    some = list(range(B)) if nb < 12 else [0, B // 2, B - 1]
    compare([t[some] for t in got], *(t[some] for t in (Q, K, V, dO)), mat, bs, None if kp is None else kp[some], FP32_TOL, False)
    rows, cols = (2 if bs == d == 32 and nb * B * H > 12 * 148 else 1), (2 if d == 32 else 1)
    want = {f"mma_fwd_kernel<{bs}, {d}, {rows}>", f"mma_bwd_row{'2' if layout == 'csr' else ''}_kernel<{bs}, {d}, {rows}>",
            f"mma_bwd_col_kernel<{bs}, {d}, {cols}, false>"}
    if nb > 11:
        want.add(f"mma_bwd_col_kernel<{bs}, {d}, {cols}, true>")
    assert all(any(w in n for n in names) for w in want), (want, names)
    assert not any("fused_" in n for n in names), names


# (bs, d, B, blocks per side, blocks per row, tensor cores): both sides of the lines between the two files (148 SMs)
@pytest.mark.parametrize("bs,d,B,nb,per,mma", [(32, 32, 14, 32, 8, False), (32, 32, 15, 32, 8, True), (32, 32, 15, 32, 3, False), (32, 32, 75, 16, 1, True),
                                               (32, 32, 2, 250, 6, False), (32, 32, 3, 180, 4, False), (32, 32, 3, 198, 4, True),
                                               (32, 64, 11, 32, 8, False), (32, 64, 12, 32, 8, True), (64, 32, 9, 16, 6, False), (64, 32, 10, 16, 6, True),
                                               (64, 64, 11, 16, 6, False), (64, 64, 12, 16, 6, True), (64, 64, 19, 16, 2, True)])
def test_fp32_calls_on_either_side_of_the_line(bs, d, B, nb, per, mma):
    from spion_b200.native import BlockSparseAttention
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(79 + nb, B, 1, L, d)
    mat = synthetic.band_random_mask(3, nb, per / nb) if per > 1 else np.eye(nb, dtype=np.uint8)
    mod = BlockSparseAttention(cfg(B, 1, L, d, bs), dtype=torch.float32)
    compare(run(mod, Q, K, V, dO, mat, None), Q, K, V, dO, mat, bs, None, FP32_TOL, False)
    names = fp32_kernels(lambda: run(mod, Q, K, V, dO, mat, None))
    assert len(names) >= 3 and all(("mma_" in n) == mma for n in names), names


@pytest.mark.parametrize("bs,d", [(32, 32), (64, 64)])
def test_fp32_tensor_core_kernels_with_values_that_are_not_finite(bs, d):
    """The parts of an infinity are NaN: rows that meet one are formed again.  A block-diagonal mask with a second block per row, so that what
    a value can reach is known: key j of block c is seen by the rows of blocks c and c - 1."""
    from spion_b200.native import BlockSparseAttention
    B, nb = 80 if bs == 32 else 40, 16
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(41, B, 1, L, d)
    mat = np.eye(nb, dtype=np.uint8) + np.roll(np.eye(nb, dtype=np.uint8), 1, axis=1)
    V[0, 0, 3 * bs + 1, 2] = float("inf")             # column 2 of O in block rows 2 and 3
    V[1, 0, 3 * bs + 1, 2] = 3.4e38                   # rounds to an infinity in bf16; finite results
    K[2, 0, 5 * bs + 3] = -1e30                       # scores far below (P = 0) or far above all others (P = 1)
    Q[3, 0, 7 * bs + 9, 0] = float("nan")             # one row
    dO[4, 0, 9 * bs + 4, 5] = float("inf")            # dV[:, 5] of the keys of blocks 9 and 10; the row of dQ; dK of both blocks
    mod = BlockSparseAttention(cfg(B, 1, L, d, bs), dtype=torch.float32)
    got = [t.detach().cpu() for t in run(mod, Q, K, V, dO, mat, None)]
    for b in range(6):
        q, k, v = (t[b, 0].double().requires_grad_(True) for t in (Q, K, V))
        rows = []
        for r in range(nb):                           # the reference's softmax: unselected keys count as score 0
            sel = torch.cat([torch.arange(c * bs, (c + 1) * bs) for c in np.flatnonzero(mat[r])])
            s = q[r * bs:(r + 1) * bs] @ k[sel].T / d ** 0.5
            m = s.detach().amax(-1, keepdim=True).clamp_min(-100.0)
            e = torch.exp(s - m)
            rows.append(e / (e.sum(-1, keepdim=True) + (L - len(sel)) * torch.exp(-m)) @ v[sel])
        out = torch.cat(rows)
        want = (out.detach(),) + torch.autograd.grad(out, (q, k, v), dO[b, 0].double())
        for name, x, y in zip(("O", "dQ", "dK", "dV"), got, want):
            x, y = x[b, 0].double(), y
            if (b == 0 and name != "O") or (b == 1 and name in ("dQ", "dK")) or (b == 2 and name == "dQ"):
                continue                              # inf - inf, or rounding multiplied by 1e30: the order of the steps decides
            fin = y.abs() < 3e38
            assert torch.equal(torch.isfinite(x), fin), (b, name, int((torch.isfinite(x) != fin).sum()))
            assert float(((x - y).abs()[fin] / y.abs()[fin].clamp_min(1.0)).max()) <= FP32_TOL, (b, name)


@pytest.mark.parametrize("bs,d", [(32, 32), (32, 64), (64, 32), (64, 64)])
@pytest.mark.parametrize("layout", ["tiles", "csr"])
@pytest.mark.parametrize("scale", [1e-30, 1e-33, 1e-36])
def test_fp32_tensor_core_kernels_with_small_values(bs, d, layout, scale):
    """V and dO so small that bf16 parts of them, of dP and of dS would fall below the smallest bf16 number.  fp32 sums of up to 1024 products:
    sqrt(1024) roundings of 2^-24 in norm."""
    B, nb = (80, 16) if bs == 32 else (48, 16)
    L = nb * bs
    Q, K, V, dO = synthetic.qkv(73, B, 1, L, d)
    mat = lines_of_every_length(nb)
    call, close = fp32_call(layout, B, 1, L, d, bs, mat, None)
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    got = [call(q, k, (V * scale).cuda()).detach()] + list(torch.autograd.grad(call(q, k, v), (q, k, v), (dO * scale).cuda()))
    close()
    want = oatt.sparse_attention(Q[:3], K[:3], V[:3], mat, bs, None, (dO * scale)[:3], dtype=torch.float64)
    want = [oatt.sparse_attention(Q[:3], K[:3], (V * scale)[:3], mat, bs, dtype=torch.float64)[0], *want[2:]]
    for name, a, b in zip(("O", "dQ", "dK", "dV"), got, want):
        err = float((a[:3].cpu().double() - b).norm() / b.norm())
        assert err <= 1024 ** 0.5 * 2.0 ** -24, f"{name}: {err:.2e}"


@pytest.mark.parametrize("bs,d,BH,nb", [(32, 64, 131071, 2), (64, 32, 65536, 2), (64, 64, 65536, 1)])      # nb 1: the full mask's kernels
def test_fp32_more_matrices_than_a_launch_takes(bs, d, BH, nb):
    """65535 groups of one or two matrices are the most that a grid has: the matrices at both sides of a slice's end."""
    from spion_b200.native import BlockSparseAttention
    L = nb * bs
    g = torch.Generator(device="cuda").manual_seed(67)
    Q, K, V, dO = (torch.randn(BH, 1, L, d, generator=g, device="cuda") for _ in range(4))
    mat = np.tril(np.ones((nb, nb), np.uint8))
    kp = synthetic.key_padding(9, 16, L).repeat((BH + 15) // 16, 1)[:BH]
    mod = BlockSparseAttention(cfg(BH, 1, L, d, bs), dtype=torch.float32, keypad=True)
    got = run(mod, Q, K, V, dO, mat, kp)
    n = -(-BH // 65535)
    end = -(-BH // n)
    some = [0, 1, 65534, 65535 % BH, end - 1, end, BH - 1]
    compare([t[some] for t in got], *(t[some].cpu() for t in (Q, K, V, dO)), mat, bs, kp[some], FP32_TOL, False)


@pytest.mark.parametrize("L,d", [(64, 64), (192, 32), (512, 32), (576, 32), (1024, 64), (1088, 32), (1856, 32)])
@pytest.mark.parametrize("padded", [False, True])
def test_dense_fp32_kernels(L, d, padded):
    """One tile, ragged softmax slices, the longest slice in registers (64 and 128 values) and one more, a slab too long for shared
    memory."""
    from spion_b200.attention import Attention
    from spion_b200.attention_cuda import CUDAAttention
    from spion_b200.attention_cuda_mask import CUDAMaskAttention
    B, H = 1, 2
    Q, K, V, dO = synthetic.qkv(31 + L, B, H, L, d)
    kp = synthetic.key_padding(2, B, L) if padded else torch.ones(B, L)
    cpp = Attention._cuda_mask_compile_module() if padded else Attention._cuda_compile_module()
    handle = cpp.init(d, L, B * H)
    mod = (CUDAMaskAttention if padded else CUDAAttention)(cfg(B, H, L, d, 32), cpp, handle)
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    out, attn = mod(q, k, v, kp.cuda())
    out.backward(dO.cuda())
    O, P, gQ, gK, gV = oatt.dense_attention(Q, K, V, kp if padded else None, dO)
    assert far(attn, P, False) <= 1e-6
    for name, a, b in zip(("O", "dQ", "dK", "dV"), (out, q.grad, k.grad, v.grad), (O, gQ, gK, gV)):
        assert far(a, b, False) <= FP32_TOL, f"{name}: {far(a, b, False):.3e}"
    cpp.destroy(handle)


@pytest.mark.parametrize("layers,L,bs,misaligned", [(1, 64, 64, False), (3, 160, 32, False), (2, 320, 64, True), (17, 128, 32, False)])
def test_discovery_of_several_layers(layers, L, bs, misaligned):
    """One cell, ragged map counts, maps that do not start on 16 bytes, more maps than one call takes: bit for bit the oracle."""
    from spion_b200 import pattern
    maps = [synthetic.structured_map(40 + i, L) for i in range(layers)]
    gpu = []
    for A in maps:
        room = torch.empty(L * L + 1, device="cuda")
        part = room[1:] if misaligned else room[:-1]
        gpu.append(part.view(L, L).copy_(A))
    mats, patterns = pattern.discover_layers(gpu, {"block_size": bs, "max_seq_len": L, "threshold": 0.8})
    assert mats.shape == (4, layers, L // bs, L // bs)
    for i, A in enumerate(maps):
        want, thresh, pooled = opat.discover_block_mask(A.numpy(), bs, 0.8, 31, 0, float_path="fixed")
        p = patterns[i]
        assert np.array_equal(p.pooled.cpu().numpy(), pooled) and float(p.thresh) == float(thresh)
        assert np.array_equal(p.mat.cpu().numpy(), want)
        assert all(np.array_equal(mats[r, i].cpu().numpy(), want.astype(np.float32)) for r in range(4))
        rp, ci, br = ocsr.block_csr(want)
        cp, ri, pos = ocsr.block_csc(want)
        for got, ref in ((p.row_ptr, rp), (p.col_idx, ci), (p.blk_row, br), (p.col_ptr, cp), (p.row_idx, ri), (p.csc_pos, pos)):
            assert np.array_equal(got.cpu().numpy(), ref)


@pytest.mark.parametrize("d,H", [(64, 2), (32, 4)])
@pytest.mark.parametrize("full_mask", [False, True])
def test_streaming_forward_with_rows_without_blocks_between_others(d, H, full_mask):
    """More matrices than stay in L2, so that the rows are walked matrix by matrix: rows with blocks follow each other directly, after
    one row without any, and after several.  Every output row against the masked softmax in fp32."""
    from spion_b200.native import BlockSparseAttention
    B, nb, bs = 84, 32, 64
    L = nb * bs
    assert 2 * B * H * L * d * 2 > 80 << 20
    mat = np.ones((nb, nb), np.uint8)
    if not full_mask:
        rng = np.random.default_rng(d)
        mat = np.zeros((nb, nb), np.uint8)
        mat[5] = 1                                           # a long row: the mask is the streaming kernel's
        for r in rng.permutation(nb)[:nb // 2]:
            mat[r, rng.choice(nb, size=rng.integers(1, 5), replace=False)] = 1
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn(B, H, L, d, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
    mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.bfloat16, return_probs=False)
    with torch.no_grad():
        out, _ = mod(q, k, v, None, torch.as_tensor(mat).cuda())
    mod.check_device_status()
    sel = torch.as_tensor(np.kron(mat, np.ones((bs, bs), np.uint8))).cuda().bool()
    others = (~sel).sum(1, keepdim=True).float()
    for b in range(B):
        e = torch.exp(q[b].float() @ k[b].float().transpose(1, 2) / d ** 0.5) * sel
        want = (e / (e.sum(-1, keepdim=True) + others)) @ v[b].float()
        assert far(out[b], want, True) <= BF16_REL, (b, far(out[b], want, True))


@pytest.mark.parametrize("d,bs", [(64, 64), (32, 64), (32, 32)])
@pytest.mark.parametrize("full", [False, True])
def test_streaming_kernels_with_penalties_of_every_kind(d, bs, full):
    """Blocks whose keys have no penalty, one penalty (small, large, negative), different ones, and a sequence of padded keys only: P is
    exp2 of scores less the penalties, so the reference takes them as an additive mask of its own."""
    from spion_b200.native import BlockSparseAttention
    B, H, nb = 3, 2, 10 if bs == 64 else 20
    L = nb * bs
    Q, K, V, dO = (t.to(torch.bfloat16) for t in synthetic.qkv(43 + d, B, H, L, d))
    mat = np.ones((nb, nb), np.uint8) if full else lines_of_every_length(nb)
    keep = torch.ones(B, L)                                  # penalty 1e6 (1 - keep)
    keep[0, 64:128] = 1 - 1.5e-6                             # one small penalty for a block
    keep[0, 128:192] = 1 + 2e-6                              # a bonus
    keep[0, 192:256] = 1 - 1e-6 * torch.arange(64) / 32      # a different one for every key
    keep[1, L - 100:] = 0                                    # a padded tail that begins inside a block
    keep[2, 0 if not full else 1:] = 0                       # nothing but padding (full mask: one key, or no score counts at all)
    mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=torch.bfloat16, keypad=True, recompute=True, return_probs=False)
    got = run(mod, Q, K, V, dO, mat, keep)
    O, _, gQ, gK, gV = oatt.sparse_attention(Q.float(), K.float(), V.float(), mat, bs, keep, dO.float(), dtype=torch.float64)
    for name, a, b in zip(("O", "dQ", "dK", "dV"), got, (O, gQ, gK, gV)):
        assert torch.isfinite(a).all()
        assert far(a[:2], b[:2], True) <= BF16_REL, f"{name}: {far(a[:2], b[:2], True):.3e}"
    if not full:                                             # unselected keys count as score 0 and leave nothing to the padded ones
        assert not got[0][2].any() and not got[3][2].any()


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("padded", [False, "keys", "soft"])
@pytest.mark.parametrize("short", [False, True])
@pytest.mark.parametrize("probs", [False, True])
def test_rebuilt_rounded_tiles_are_the_stored_ones(d, padded, short, probs):
    """Gradients without stored tiles, bit for bit: rows of up to four blocks (normalised after a rounding) and longer ones (before it), masks
    of short rows only, blocks with no, one and different penalties (soft: penalties that leave P above zero), odd last pairs, lines without
    blocks."""
    from spion_b200.native import BlockSparseAttention
    B, H, nb = 2, 3, 11
    L = nb * 64
    Q, K, V, dO = (t.to(torch.bfloat16) for t in synthetic.qkv(47 + d, B, H, L, d))
    mat = lines_of_every_length(nb)
    if short:
        mat = np.triu(mat, -3)
    kp = synthetic.key_padding(5, B, L) if padded else None
    if padded == "soft":
        kp[0] = 1 - 1e-6 * torch.rand(L, generator=torch.Generator().manual_seed(71)) * 3
        kp[0, 128:192] = 1 - 1.5e-6
    got = []
    for recompute in (None, False):
        mod = BlockSparseAttention(cfg(B, H, L, d, 64), dtype=torch.bfloat16, keypad=bool(padded), recompute=recompute, return_probs=probs)
        mod.set_mask(torch.as_tensor(mat).cuda())
        if recompute is None:                                # what calls with probabilities, and small ones at head_dim 32, do
            mod.recompute, mod._ctx.rounded = False, True
        n0 = mod.launch_count()
        q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
        out, _ = mod(q, k, v, None if kp is None else kp.cuda())
        got.append((out,) + torch.autograd.grad(out, (q, k, v), dO.cuda()))
        mod.check_device_status()
        assert mod.launch_count() - n0 == 3                  # forward, rows, columns
    for name, a, b in zip(("O", "dQ", "dK", "dV"), *got):
        assert torch.equal(a, b), f"{name}: {far(a, b, True):.3e}"
    compare(got[0], Q, K, V, dO, mat, 64, kp, BF16_REL, True)


# (d, padded, P returned, matrices, blocks per side, blocks per row, rebuilt): both sides of the lines between rebuilt and stored rounded tiles
@pytest.mark.parametrize("d,padded,probs,BH,nb,per,rebuilt",
                         [(32, False, False, 31, 8, 2, False), (32, False, False, 32, 8, 2, True), (64, False, True, 17, 10, 3, False), (64, False, True, 18, 10, 3, True),
                          (32, True, False, 102, 10, 4, False), (32, True, False, 103, 10, 4, True), (32, True, True, 410, 10, 4, False), (64, True, True, 327, 10, 5, False),
                          (64, True, True, 328, 10, 5, True), (32, True, True, 34, 12, 10, False), (32, True, True, 35, 12, 10, True)])
def test_rounded_tiles_are_rebuilt_or_stored(d, padded, probs, BH, nb, per, rebuilt):
    from torch.profiler import ProfilerActivity, profile

    from spion_b200.native import BlockSparseAttention
    L = nb * 64
    Q, K, V, dO = (t.to(torch.bfloat16) for t in synthetic.qkv(83 + d, BH, 1, L, d))
    mat = np.zeros((nb, nb), np.uint8)
    for r in range(nb):
        mat[r, [(r + i) % nb for i in range(per)]] = 1
    kp = synthetic.key_padding(5, BH, L) if padded else None
    got = []
    for recompute in (None, False):
        mod = BlockSparseAttention(cfg(BH, 1, L, d, 64), dtype=torch.bfloat16, keypad=padded, recompute=recompute, return_probs=probs)
        run(mod, Q, K, V, dO, mat, kp)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            got.append(run(mod, Q, K, V, dO, mat, kp))
        names = {e.name for e in prof.events()}
        assert any("k_bwd_stream" in n for n in names) == (rebuilt and recompute is None), names
        assert any("k_bwd_row" in n for n in names) == (not rebuilt or recompute is False), names
    for name, a, b in zip(("O", "dQ", "dK", "dV"), *got):
        assert torch.equal(a, b), f"{name}: {far(a, b, True):.3e}"


@pytest.mark.parametrize("d", [32, 64])
def test_gradients_read_the_probabilities_that_a_hook_hands_back(d):
    """A hook on saved tensors that gives halved probabilities to the backward halves dV: exact in bf16."""
    from spion_b200.native import BlockSparseAttention
    B, H, nb = 1, 2, 5
    L = nb * 64
    Q, K, V, dO = (t.to(torch.bfloat16).cuda() for t in synthetic.qkv(53 + d, B, H, L, d))
    mod = BlockSparseAttention(cfg(B, H, L, d, 64), dtype=torch.bfloat16, keypad=False, return_probs=True)
    mod.set_mask(torch.as_tensor(np.triu(np.ones((nb, nb), dtype=np.int64))).cuda())
    got = []
    for factor in (1.0, 0.5):
        def hand_back(t, factor=factor):
            return t * factor if t.dtype == torch.bfloat16 and t.numel() == B * H * mod.nnz else t
        q, k, v = (t.clone().requires_grad_(True) for t in (Q, K, V))
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, hand_back):
            out, _ = mod(q, k, v, None)
        got.append(torch.autograd.grad(out, v, dO)[0])
    assert torch.equal(got[1], got[0] * 0.5)


@pytest.mark.parametrize("dtype,d,bs", [(torch.float32, 64, 64), (torch.float32, 32, 32), (torch.bfloat16, 64, 64), (torch.bfloat16, 32, 64)])
def test_kernels_that_start_beside_the_one_before_under_capture(dtype, d, bs):
    """Backward kernels that are placed before the kernel ahead of them has ended (fp32: columns with and without a full one; bf16: rows, columns), in
    a CUDA graph replayed on other values, the bits of eager calls."""
    from spion_b200.native import BlockSparseAttention
    B, H, nb = 1, 30, 33
    L = nb * bs if bs == 64 else nb * 64
    nb = L // bs
    rng = np.random.default_rng(61)
    mat = (rng.random((nb, nb)) < 0.1).astype(np.int64)
    np.fill_diagonal(mat, 1)
    mat[:, 5] = 1
    mod = BlockSparseAttention(cfg(B, H, L, d, bs), dtype=dtype, keypad=False, return_probs=False)
    mod.set_mask(torch.as_tensor(mat).cuda())
    static = [torch.empty(B, H, L, d, dtype=dtype, device="cuda").requires_grad_(i < 3) for i in range(4)]

    def step():
        out = mod(*static[:3], None)[0]
        return (out,) + torch.autograd.grad(out, static[:3], static[3])

    def load(seed):
        with torch.no_grad():
            for s, t in zip(static, synthetic.qkv(seed, B, H, L, d)):
                s.copy_(t.to(dtype))

    load(3)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for seed in (4, 5):
        load(seed)
        for _ in range(3):
            graph.replay()
        replayed = [t.clone() for t in got]
        for a, b in zip(replayed, step()):
            assert torch.equal(a, b)
    mod.check_device_status()
