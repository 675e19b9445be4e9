"""GPU tests of the linear-layer kernels (csrc/linear.cu) and of the one-node attention layer, against fp64 products."""
import ctypes

import pytest
import torch

from spion_b200 import _lib
from spion_b200._lib import Tokens, check, lib

pytestmark = pytest.mark.gpu


def _tokens(ts, heads=0, d=0, L=0):
    t = Tokens()
    t.count, t.is_bf16, t.heads, t.head_dim, t.seq_len = len(ts), int(ts[0].dtype == torch.bfloat16), heads, d, L
    for i, x in enumerate(ts):
        t.ptr[i] = x.data_ptr()
    t.cols = heads * d if heads else ts[0].shape[-1]
    return t


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# tokens per sequence around the 64 / 128-token tiles; widths with a partial 64-feature chunk (32, 96), one and three stacked
# matrices, contractions of several chunks and (fp32, 384) one that takes several launches
@pytest.mark.parametrize("B,L,H,d,K,nw", [(1, 1, 1, 32, 32, 1), (1, 129, 2, 32, 64, 3), (3, 63, 3, 32, 96, 3), (2, 191, 4, 32, 128, 3),
                                          (1, 20000, 2, 32, 64, 1), (2, 100, 3, 64, 192, 1), (1, 300, 4, 64, 256, 3)])
@pytest.mark.parametrize("mode", ["bf16", "bf16_x", "fp32"])
@pytest.mark.parametrize("split", [False, True])
def test_linear_kernels(B, L, H, d, K, nw, mode, split):
    fp32 = int(mode == "fp32")
    N1, T = H * d, B * L
    N = nw * N1
    if not lib.spion_linear_supported(K, N, fp32) or (mode == "bf16_x" and nw == 3 and N1 % 64):
        pytest.skip("width not served")
    g = torch.Generator(device="cuda").manual_seed(T + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    P = ctypes.c_void_p
    st = P(torch.cuda.current_stream().cuda_stream)
    yt = torch.float32 if fp32 else torch.bfloat16
    X = rnd(T, K).to(torch.bfloat16 if mode == "bf16_x" else torch.float32)
    Ws, bs = [rnd(N1, K) for _ in range(nw)], [rnd(N1) for _ in range(nw)]
    ptrs = lambda ts: (P * 3)(*([t.data_ptr() for t in ts] + [None] * (3 - len(ts))))
    shape, lay = ((B, H, L, d), (H, d, L)) if split else ((T, N1), (0, 0, 0))
    cat = lambda ts: torch.cat([(t.permute(0, 2, 1, 3).reshape(T, N1) if split else t) for t in ts], 1).double()
    Ys = [torch.full(shape, 7.0, dtype=yt, device="cuda") for _ in range(nw)]
    dYs = [rnd(*shape).to(yt) for _ in range(nw)]
    dX = torch.full((T, K), 7.0, dtype=X.dtype, device="cuda")
    dW, db = torch.full((N, K), 7.0, device="cuda"), torch.full((N,), 7.0, device="cuda")
    ws = torch.empty(lib.spion_linear_workspace_floats(T, K, N, fp32), device="cuda")
    tx, ty, td, tdx = _tokens([X]), _tokens(Ys, *lay), _tokens(dYs, *lay), _tokens([dX])
    ref = ctypes.byref
    check(lib.spion_linear_forward(ref(tx), ptrs(Ws), ptrs(bs), nw, fp32, ref(ty), None, T, K, N, st))
    check(lib.spion_linear_backward_input(ref(td), ptrs(Ws), nw, fp32, None, ref(tdx), T, K, N, st))
    check(lib.spion_linear_backward_weight(ref(td), ref(tx), fp32, P(dW.data_ptr()), P(db.data_ptr()), P(ws.data_ptr()), T, K, N, st))
    torch.cuda.synchronize()
    assert lib.spion_linear_status(1) == 0
    W, b, dY = torch.cat(Ws).double(), torch.cat(bs).double(), cat(dYs)
    # bf16: operands and result carry a relative error of 2^-9 each (uniformly distributed rounding: 2^-9 / sqrt(3) rms per
    # factor).  fp32: rounding of the result plus the fp32 additions of the contraction, a few 2^-24.
    tol = 5e-7 if fp32 else 5e-3
    assert _rel(cat(Ys), X.double() @ W.t() + b) < tol
    assert _rel(dX, dY @ W) < tol
    assert _rel(dW, dY.t() @ X.double()) < (2e-6 if fp32 else tol)
    assert _rel(db, dY.sum(0)) < 2e-6


# bf16 tokens, more than 148 tiles of 128 (read through tensor maps) and fewer: sequences of 64-token boxes that end at and in the
# middle of a tile, row-major tails of 56 and 1 tokens, heads of 32 and 64, one to three matrices; widths and lengths that are copied
# sequences of whole half-tiles (boxes of 32 tokens): one half, an odd number of them, several tiles per CTA; boxes of 32 and 64 features, rows
# of one head and parts of longer rows
@pytest.mark.parametrize("B,L,H,d,K,nw", [(1, 32, 1, 64, 64, 1), (3, 32, 2, 32, 96, 3), (5, 96, 3, 64, 192, 3), (2, 64, 1, 128, 160, 1), (70, 320, 2, 64, 64, 3),
                                          (100, 320, 2, 32, 64, 1)])
def test_fp32_linear_kernels_on_whole_boxes(B, L, H, d, K, nw):
    for split in (False, True):
        test_linear_kernels(B, L, H, d, K, nw, "fp32", split)


@pytest.mark.parametrize("B,L,H,d,N,nw", [(149, 128, 2, 32, 64, 1), (101, 192, 2, 32, 64, 3), (300, 64, 4, 32, 96, 1), (61, 320, 1, 64, 64, 3),
                                          (101, 192, 2, 64, 192, 1), (1, 19000, 2, 32, 64, 3), (1, 19073, 1, 64, 128, 1),
                                          (40, 1984, 2, 32, 64, 3), (101, 192, 3, 32, 64, 1), (120, 160, 2, 32, 64, 3),
                                          (3, 192, 2, 32, 64, 3), (1, 129, 2, 32, 64, 1)])
@pytest.mark.parametrize("split", [False, True])
def test_linear_kernels_on_bf16_tokens(B, L, H, d, N, nw, split):
    T, K = B * L, H * d
    g = torch.Generator(device="cuda").manual_seed(T + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    P, ref = ctypes.c_void_p, ctypes.byref
    st = P(torch.cuda.current_stream().cuda_stream)
    shape, lay = ((B, H, L, d), (H, d, L)) if split else ((T, K), (0, 0, 0))
    flat = lambda t: (t.permute(0, 2, 1, 3).reshape(T, K) if split else t).double()
    A = [rnd(*shape).to(torch.bfloat16) for _ in range(nw)]          # forward (nw == 1) and input gradient of nw stacked layers
    ptrs = lambda ts: (P * 3)(*([t.data_ptr() for t in ts] + [None] * (3 - len(ts))))
    ta = _tokens(A, *lay)
    if nw == 1:                                                      # the output projection: tokens in, rows out
        W, b, Y, dY = rnd(N, K), rnd(N), torch.full((T, N), 7.0, device="cuda", dtype=torch.bfloat16), rnd(T, N).to(torch.bfloat16)
        ty, tdy = _tokens([Y]), _tokens([dY])
        check(lib.spion_linear_forward(ref(ta), ptrs([W]), ptrs([b]), 1, 0, ref(ty), None, T, K, N, st))
        dW, db = torch.full((N, K), 7.0, device="cuda"), torch.full((N,), 7.0, device="cuda")
        ws = torch.empty(lib.spion_linear_workspace_floats(T, K, N, 0), device="cuda")
        check(lib.spion_linear_backward_weight(ref(tdy), ref(ta), 0, P(dW.data_ptr()), P(db.data_ptr()), P(ws.data_ptr()), T, K, N, st))
        torch.cuda.synchronize()
        assert _rel(Y, flat(A[0]) @ W.double().t() + b.double()) < 5e-3
        assert _rel(dW, dY.double().t() @ flat(A[0])) < 2e-6          # exact products of bf16 values, fp32 sums
    else:                                                            # gradients of three stacked layers: rows of N features in
        Ws = [rnd(K, N) for _ in range(nw)]
        X, dX = rnd(T, N).to(torch.bfloat16), torch.full((T, N), 7.0, device="cuda")
        tx, tdx = _tokens([X]), _tokens([dX])
        check(lib.spion_linear_backward_input(ref(ta), ptrs(Ws), nw, 0, None, ref(tdx), T, N, nw * K, st))
        dW, db = torch.full((nw * K, N), 7.0, device="cuda"), torch.full((nw * K,), 7.0, device="cuda")
        ws = torch.empty(lib.spion_linear_workspace_floats(T, N, nw * K, 0), device="cuda")
        check(lib.spion_linear_backward_weight(ref(ta), ref(tx), 0, P(dW.data_ptr()), P(db.data_ptr()), P(ws.data_ptr()), T, N, nw * K, st))
        torch.cuda.synchronize()
        dY = torch.cat([flat(t) for t in A], 1)
        assert _rel(dX, dY @ torch.cat(Ws).double()) < 5e-3
        assert _rel(dW, dY.t() @ X.double()) < 2e-6
    assert lib.spion_linear_status(1) == 0
    assert _rel(db, (dY.double() if nw == 1 else dY).sum(0)) < 2e-6


# The other results of bf16 tokens read through tensor maps (more than 148 tiles of 128).  W enters the products rounded to bf16, the sums are
# fp32: results rounded to bf16 as the reference's are differ where such a sum (error about 2^-20) falls beside a tie, in at most a few
# of a hundred elements, by 2^-8 each: less than 1e-3 in norm.
def _bf(t):
    return t.to(torch.bfloat16).double()


@pytest.mark.parametrize("B,L,H,d,N", [(101, 192, 2, 32, 64), (61, 320, 1, 64, 64), (101, 192, 2, 64, 192), (40, 1984, 4, 32, 96)])
@pytest.mark.parametrize("split", [False, True])
def test_bf16_gradient_of_three_layers(B, L, H, d, N, split):
    """Each layer's gradient rounded, added in bf16 from the last to the first."""
    T, K = B * L, H * d
    g = torch.Generator(device="cuda").manual_seed(T + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    P, st = ctypes.c_void_p, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    shape, lay = ((B, H, L, d), (H, d, L)) if split else ((T, K), (0, 0, 0))
    dY = [rnd(*shape).to(torch.bfloat16) for _ in range(3)]
    Ws, dX = [rnd(K, N) for _ in range(3)], torch.full((T, N), 7.0, device="cuda", dtype=torch.bfloat16)
    check(lib.spion_linear_backward_input(ctypes.byref(_tokens(dY, *lay)), (P * 3)(*[w.data_ptr() for w in Ws]), 3, 0, None,
                                          ctypes.byref(_tokens([dX])), T, N, 3 * K, st))
    torch.cuda.synchronize()
    assert lib.spion_linear_status(1) == 0
    a, b, c = (_bf((t.permute(0, 2, 1, 3).reshape(T, K) if split else t).double() @ _bf(w)) for t, w in zip(dY, Ws))
    assert _rel(dX, _bf(_bf(c + b) + a)) < 1e-3


@pytest.mark.parametrize("T,K,N", [(19073, 64, 128), (19456, 96, 64), (75776, 128, 256)])
def test_gelu_on_bf16_tokens(T, K, N):
    """Forward with the activation, and the gradient through it."""
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    P, st = ctypes.c_void_p, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptrs = lambda t: (P * 3)(t.data_ptr(), None, None)
    X, W, b = rnd(T, K).to(torch.bfloat16), rnd(N, K) / K ** 0.5, rnd(N)
    Y, G = (torch.full((T, N), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    check(lib.spion_linear_forward(ctypes.byref(_tokens([X])), ptrs(W), ptrs(b), 1, 0, ctypes.byref(_tokens([Y])), P(G.data_ptr()), T, K, N, st))
    dY, V = rnd(T, K).to(torch.bfloat16), rnd(K, N) / N ** 0.5           # of a second layer [K, N] behind the activation
    dX = torch.full((T, N), 7.0, device="cuda", dtype=torch.bfloat16)
    check(lib.spion_linear_backward_input(ctypes.byref(_tokens([dY])), ptrs(V), 1, 0, P(Y.data_ptr()), ctypes.byref(_tokens([dX])), T, N, K, st))
    torch.cuda.synchronize()
    assert lib.spion_linear_status(1) == 0
    assert _rel(Y, _bf(X.double() @ _bf(W).t() + _bf(b))) < 1e-3
    h = Y.double().requires_grad_()
    act = torch.nn.functional.gelu(h)
    assert _rel(G, _bf(act.detach())) < 1e-3
    slope, = torch.autograd.grad(act.sum(), h)
    assert _rel(dX, _bf(_bf(dY.double() @ _bf(V)) * slope)) < 1e-3


@pytest.mark.parametrize("B,L,heads,fp32", [(1, 1, 1, 0), (3, 127, 2, 0), (2, 4096, 3, 1), (150, 160, 2, 0), (7, 33, 8, 1)])
def test_projections_with_the_penalties_of_padded_keys(B, L, heads, fp32):
    """The penalties that the projections' kernel writes are spion_expand_keypad's, and its outputs those without them."""
    P = ctypes.c_void_p
    st = P(torch.cuda.current_stream().cuda_stream)
    T, K, N = B * L, 64, 96
    X, W, b = torch.randn(T, K, device="cuda"), torch.randn(N, K, device="cuda"), torch.randn(N, device="cuda")
    yt = torch.float32 if fp32 else torch.bfloat16
    Y, Z = (torch.full((T, N), 7.0, dtype=yt, device="cuda") for _ in range(2))
    mask = (torch.rand(B, L, device="cuda") < 0.7).float()
    pen, want = (torch.full((B * heads, L), -1.0, device="cuda") for _ in range(2))
    one, ref = lambda t: (P * 3)(t.data_ptr(), None, None), ctypes.byref
    check(lib.spion_linear_forward_keypad(ref(_tokens([X])), one(W), one(b), 1, fp32, ref(_tokens([Y])), None, None, T, K, N, P(mask.data_ptr()), B, heads, L,
                                          P(pen.data_ptr()), st))
    check(lib.spion_linear_forward(ref(_tokens([X])), one(W), one(b), 1, fp32, ref(_tokens([Z])), None, T, K, N, st))
    check(lib.spion_expand_keypad(P(mask.data_ptr()), B, heads, L, P(want.data_ptr()), st))
    assert torch.equal(pen, want) and torch.equal(Y, Z)
    assert lib.spion_linear_forward_keypad(ref(_tokens([X])), one(W), one(b), 1, fp32, ref(_tokens([Y])), None, None, T, K, N, P(mask.data_ptr()), B + 1, heads, L,
                                           P(pen.data_ptr()), st) != 0


def test_penalties_up_to_the_largest_count():
    """2^31 - 2 penalties, two less than an int holds: what a thread would write next lies beyond that."""
    P = ctypes.c_void_p
    B, L, heads = 62, 49981, 693                                 # B L heads = 2^31 - 2
    T, K, N = B * L, 32, 32
    assert T * heads == 2 ** 31 - 2
    X, W, b = torch.zeros(T, K, dtype=torch.bfloat16, device="cuda"), torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
    Y = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    mask = (torch.rand(B, L, device="cuda") < 0.7).float()
    pen = torch.full((T * heads + 65536,), -1.0, device="cuda")
    one, ref = lambda t: (P * 3)(t.data_ptr(), None, None), ctypes.byref
    check(lib.spion_linear_forward_keypad(ref(_tokens([X])), one(W), one(b), 1, 0, ref(_tokens([Y])), None, None, T, K, N, P(mask.data_ptr()), B, heads, L,
                                          P(pen.data_ptr()), P(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert bool((pen[T * heads:] == -1.0).all())
    rows = pen[:T * heads].view(B, heads, L)
    for i in range(B):
        assert bool((rows[i] == 1e6 * (1 - mask[i])).all())


@pytest.mark.parametrize("T,K,N", [(19000, 64, 128), (20001, 32, 96), (300, 64, 64)])
def test_gelu_of_every_bf16_number(T, K, N):
    """Activation and its derivative by table, inside and outside of its range (subnormals, infinities and NaN too), the outputs through tiles in
    shared memory (more than 148 tiles of 128 tokens) and from registers: the same bits as the formulas evaluated for every bf16 number, which
    are the framework's GELU to two roundings of fp32 and one of bf16."""
    P = ctypes.c_void_p
    st = P(torch.cuda.current_stream().cuda_stream)
    ref = ctypes.byref
    g = torch.Generator(device="cuda").manual_seed(T)
    bits = torch.randint(0, 65536, (T, N), generator=g, device="cuda", dtype=torch.int32)
    bits[:T // 2] = (torch.randn(T // 2, N, generator=g, device="cuda").bfloat16().view(torch.int16).int()) & 0xffff
    h = bits.to(torch.int16).view(torch.bfloat16).contiguous()
    # derivative: dX = (dY V) * gelu'(h), dY V = a column of ones by an all-ones first feature
    dY, V = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16), torch.zeros(K, N, device="cuda")
    dY[:, 0] = 1
    V[0] = 1
    dX = torch.empty(T, N, device="cuda", dtype=torch.bfloat16)
    one = lambda t: (P * 3)(t.data_ptr(), None, None)
    check(lib.spion_linear_backward_input(ref(_tokens([dY])), one(V), 1, 0, P(h.data_ptr()), ref(_tokens([dX])), T, N, K, st))
    x = h.double()
    want = 0.5 * (1 + torch.erf(x / 2 ** 0.5)) + x * torch.exp(-0.5 * x * x) / (2 * torch.pi) ** 0.5
    ok = torch.isfinite(x)
    err = (dX.double() - want).abs()
    assert bool((err[ok] <= 2 ** -8 * want[ok].abs() + 1e-6).all())
    assert bool(torch.isnan(dX[torch.isnan(x)]).all())
    # activation: h again from a weight of ones, one bf16 number per token
    col = h[:, :1].contiguous()
    X, W, b = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16), torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
    X[:, :1] = torch.where(torch.isfinite(col), col, 0)
    W[:, 0] = 1
    Y, G = (torch.empty(T, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    check(lib.spion_linear_forward(ref(_tokens([X])), one(W), one(b), 1, 0, ref(_tokens([Y])), P(G.data_ptr()), T, K, N, st))
    y = X[:, :1].double().expand(T, N)
    assert bool(((Y.double() - y).abs() <= 1e-37).all())           # subnormals may be flushed
    want = 0.5 * y * (1 + torch.erf(y / 2 ** 0.5))
    assert bool(((G.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * y.abs().clamp(max=10) + 1e-37).all())
    assert lib.spion_linear_status(1) == 0


@pytest.mark.parametrize("native,dtype,bs,L,dense", [(True, "bf16", 64, 192, False), (True, "bf16", 64, 128, True),
                                                     (True, "fp32", 32, 160, False), (False, "fp32", 32, 96, False)])
def test_attention_layer_in_one_node_equals_its_stages(native, dtype, bs, L, dense):
    """The same layer with a forward hook on one projection runs stage by stage: same results, same gradients."""
    from contextlib import nullcontext

    from spion_b200.attention import Attention
    B, H, d = 3, 2, 32
    cfg = {"head_dim": d, "num_head": H, "max_seq_len": L, "batch_size": B, "block_size": bs, "transformer_dim": H * d,
           "task": "lra-text", "native": native, "dtype": dtype}
    torch.manual_seed(1)
    layer = Attention(cfg).cuda()
    mat = None
    if not dense:
        layer.reconstruct_for_blocksparse(cfg)
        mat = (torch.rand(L // bs, L // bs, device="cuda") < 0.5).float()
        mat.fill_diagonal_(1)
    x = torch.randn(B, L, H * d, device="cuda", requires_grad=True)
    mask = torch.ones(B, L, device="cuda")
    mask[1, L // 2:] = 0
    amp = torch.autocast("cuda", dtype=torch.bfloat16) if dtype == "bf16" else nullcontext()
    outs = []
    for hooked in (False, True):
        h = layer.W_k.register_forward_hook(lambda m, i, o: None) if hooked else None
        with amp:
            out, _ = layer(x, mask, mat)
        g = torch.autograd.grad(out, [x] + list(layer.parameters()), torch.ones_like(out))
        outs.append([out, *g])
        if h:
            h.remove()
    # bf16: the stages round dX of each projection to bf16 and add; the node adds first (two roundings of 2^-9 apart)
    tol = 2e-2 if dtype == "bf16" else 1e-5
    for a, b in zip(*outs):
        assert a.shape == b.shape and a.dtype == b.dtype
        err = float((a.double() - b.double()).norm())
        assert err <= tol * float(b.double().norm()) + 1e-6, (err, float(b.double().norm()))


@pytest.mark.parametrize("native,bs,L,H,d,keypad", [(True, 32, 160, 2, 32, True), (True, 64, 320, 3, 64, False), (False, 32, 96, 1, 32, False),
                                                    (False, 64, 192, 4, 64, True)])
def test_dense_fp32_layer_in_one_node_equals_its_stages(native, bs, L, H, d, keypad):
    """Dense attention in fp32: outputs, map and gradients of the node are those of the stages (fp32 sums of at most 960 terms in another
    order), and the gradient of the key projection's bias, which is zero but for the rounding of the stages, is the same bits."""
    from spion_b200.attention import Attention
    B = 5
    cfg = {"head_dim": d, "num_head": H, "max_seq_len": L, "batch_size": B, "block_size": bs, "transformer_dim": H * d,
           "task": "lra-text" if keypad else "lra-image", "native": native, "dtype": "fp32"}
    torch.manual_seed(3)
    layer = Attention(cfg).cuda()
    x = torch.randn(B, L, H * d, device="cuda", requires_grad=True)
    do = torch.randn(B, L, H * d, device="cuda")
    mask = torch.ones(B, L, device="cuda")
    mask[1, L // 2:] = 0
    names = ["x"] + [n for n, _ in layer.named_parameters()]
    runs = []
    for hooked in (False, True):
        h = layer.W_k.register_forward_hook(lambda m, i, o: None) if hooked else None
        out, attn = layer(x, mask, None)
        if not hooked:
            assert out.grad_fn.name() == "SparseAttentionLayerBackward"
        runs.append([out, attn if torch.is_tensor(attn) else out, *torch.autograd.grad(out, [x] + list(layer.parameters()), do)])
        if h:
            h.remove()
    assert torch.equal(runs[0][1], runs[1][1]) or native
    for n, a, b in zip(["out", "attn"] + names, *runs):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride(), n
        if n == "W_k.bias":
            assert torch.equal(a, b)
        else:
            assert float((a.double() - b.double()).norm()) <= 1e-5 * float(b.double().norm()), n


@pytest.mark.parametrize("dim,hidden", [(1024, 256), (992, 1024), (96, 992)])
def test_feed_forward_block_of_wide_layers(dim, hidden):
    """The same at the widths that leave the activation's table no room, forward or backward."""
    from spion_b200._ops import ops
    torch.manual_seed(0)
    l1, l2 = torch.nn.Linear(dim, hidden).cuda(), torch.nn.Linear(hidden, dim).cuda()
    x = torch.randn(2, 77, dim, device="cuda").bfloat16().requires_grad_(True)
    go = torch.randn(2, 77, dim, device="cuda").bfloat16()
    ps = [x, l1.weight, l1.bias, l2.weight, l2.bias]
    assert ops.mlp_supported(*ps)
    y = ops.mlp(*ps)
    got = [y, *torch.autograd.grad(y, ps, go)]
    pd = [t.detach().double().requires_grad_(True) for t in ps]
    yd = torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(pd[0], pd[1], pd[2])), pd[3], pd[4])
    for a, b in zip(got, [yd, *torch.autograd.grad(yd, pd, go.double())]):
        assert _rel(a.detach(), b.detach()) < 1.5e-2          # a chain of up to four roundings to bf16


def test_feed_forward_block():
    """Linear -> GELU -> Linear with the activation inside the kernels, against the framework's operators in bf16."""
    from spion_b200._ops import ops
    torch.manual_seed(0)
    l1, l2 = torch.nn.Linear(64, 128).cuda(), torch.nn.Linear(128, 64).cuda()
    x = torch.randn(2, 77, 64, device="cuda").bfloat16().requires_grad_(True)
    go = torch.randn(2, 77, 64, device="cuda").bfloat16()
    ps = [x, l1.weight, l1.bias, l2.weight, l2.bias]
    y = ops.mlp(x, l1.weight, l1.bias, l2.weight, l2.bias)
    got = [y, *torch.autograd.grad(y, ps, go)]
    pd = [t.detach().double().requires_grad_(True) for t in ps]
    yd = torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(pd[0], pd[1], pd[2])), pd[3], pd[4])
    want = [yd, *torch.autograd.grad(yd, pd, go.double())]
    for a, b in zip(got, want):
        assert _rel(a.detach(), b.detach()) < 1.5e-2          # a chain of up to four roundings to bf16


# widths at which the weights leave no room for the activation's table, few tiles and many; the widest with it
@pytest.mark.parametrize("T,K,N", [(300, 1024, 64), (300, 992, 96), (20001, 1024, 1024), (19100, 992, 256), (300, 960, 1024), (19100, 960, 64)])
def test_gelu_of_wide_contractions(T, K, N):
    assert lib.spion_linear_supported(K, N, 0) and lib.spion_linear_supported(N, K, 0)
    test_gelu_on_bf16_tokens(T, K, N)


def test_gelu_by_table_and_by_functions_are_the_same_bits():
    """Activation and derivative of all 65536 numbers of bf16, from kernels that look them up (64 features) and that form them (1024).
    (How far they are from the exact ones: test_gelu_of_every_bf16_number.)"""
    P, st = ctypes.c_void_p, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    one, ref = lambda t: (P * 3)(t.data_ptr(), None, None), ctypes.byref
    every = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16)
    acts, slopes = [], []
    for K in (64, 1024):
        N = 64
        h = every.view(-1, N).view(torch.bfloat16)
        T = h.shape[0]
        # derivative: a row of ones times a weight of ones in one feature
        dY, V, dX = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16), torch.zeros(K, N, device="cuda"), torch.empty_like(h)
        dY[:, 0] = 1
        V[0] = 1
        check(lib.spion_linear_backward_input(ref(_tokens([dY])), one(V), 1, 0, P(h.data_ptr()), ref(_tokens([dX])), T, N, K, st))
        slopes.append(dX.flatten())
        # activation: a number per token, in its first feature (an infinity in another column would be a NaN in this one)
        T = 65536
        X, W, b = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16), torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
        X[:, 0] = every.view(torch.bfloat16)
        W[:, 0] = 1
        Y, G = (torch.empty(T, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        check(lib.spion_linear_forward(ref(_tokens([X])), one(W), one(b), 1, 0, ref(_tokens([Y])), P(G.data_ptr()), T, K, N, st))
        assert bool((Y.view(torch.int16) == Y[:, :1].view(torch.int16)).all()) and bool((G.view(torch.int16) == G[:, :1].view(torch.int16)).all())
        acts.append((Y[:, 0], G[:, 0]))
    x = every.view(torch.bfloat16)
    same = lambda a, b: bool(((a.view(torch.int16) == b.view(torch.int16)) | (torch.isnan(a) & torch.isnan(b))).all())
    assert same(acts[0][0], acts[1][0]) and same(acts[0][1], acts[1][1]) and same(*slopes)
    normal = torch.isfinite(x) & (x.abs() >= 2.0 ** -126)
    assert torch.equal(acts[0][0][normal], x[normal])
    # a negative infinity times zero is a NaN, in the formulas as in the framework's
    assert bool(torch.isnan(acts[0][1][torch.isnan(x)]).all()) and float(acts[0][1][x == float("inf")]) == float("inf")
    assert bool(torch.isnan(acts[0][1][x == float("-inf")])) and bool(torch.isnan(slopes[0][torch.isinf(x) | torch.isnan(x)]).all())
    assert lib.spion_linear_status(1) == 0


@pytest.mark.parametrize("T,K,N", [(1 << 20, 64, 64), (1 << 18, 64, 192), (1 << 17, 256, 1024)])
def test_weight_gradient_of_many_tokens(T, K, N):
    """fp32: the error does not grow with the number of tokens.  Operands of one sign, so that the result is the sum of magnitudes: at
    most 40 truncated steps of 2^-23 per accumulator, whatever T."""
    from spion_b200.layernorm import BiasGradLinear
    lin = BiasGradLinear(K, N).cuda()
    g = torch.Generator(device="cuda").manual_seed(T)
    x, go = torch.rand(T, K, generator=g, device="cuda"), torch.rand(T, N, generator=g, device="cuda")
    dw, db = torch.autograd.grad(lin(x), [lin.weight, lin.bias], go)
    assert lib.spion_linear_supported(K, N, 1)
    assert _rel(dw, go.double().t() @ x.double()) < 40 * 2.0 ** -23
    assert _rel(db, go.double().sum(0)) < 2e-6


@pytest.mark.parametrize("split", [False, True])
def test_values_that_are_not_finite_in_bf16(split):
    """fp32: infinities, NaN and numbers above the largest of bf16 give what an fp32 product gives; everything else is as without them."""
    B, L, H, d, K, nw = 2, 150, 2, 32, 96, 3
    T, N1 = B * L, H * d
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: 0.1 * torch.randn(*s, generator=g, device="cuda")       # no product of a large number overflows
    P = ctypes.c_void_p
    st = P(torch.cuda.current_stream().cuda_stream)
    X, Ws, bs = rnd(T, K), [rnd(N1, K) for _ in range(nw)], [rnd(N1) for _ in range(nw)]
    shape, lay = ((B, H, L, d), (H, d, L)) if split else ((T, N1), (0, 0, 0))
    dYs = [rnd(*shape) for _ in range(nw)]
    big, inf, nan = 3.4e38, float("inf"), float("nan")
    X[3, 5], X[140, 95], X[141, 0], X[290, 64] = big, inf, -inf, nan
    Ws[1][7, 33] = -inf
    flat = [t.view(-1) for t in dYs]
    flat[0][11], flat[1][4000], flat[2][9000] = inf, big, nan
    ptrs = lambda ts: (P * 3)(*([t.data_ptr() for t in ts] + [None] * (3 - len(ts))))
    cat = lambda ts: torch.cat([(t.permute(0, 2, 1, 3).reshape(T, N1) if split else t) for t in ts], 1).double()
    Ys, dX = [torch.empty(shape, device="cuda") for _ in range(nw)], torch.empty(T, K, device="cuda")
    N = nw * N1
    dW, db = torch.empty(N, K, device="cuda"), torch.empty(N, device="cuda")
    ws = torch.empty(lib.spion_linear_workspace_floats(T, K, N, 1), device="cuda")
    tx, ty, td, tdx = _tokens([X]), _tokens(Ys, *lay), _tokens(dYs, *lay), _tokens([dX])
    ref = ctypes.byref
    check(lib.spion_linear_forward(ref(tx), ptrs(Ws), ptrs(bs), nw, 1, ref(ty), None, T, K, N, st))
    check(lib.spion_linear_backward_input(ref(td), ptrs(Ws), nw, 1, None, ref(tdx), T, K, N, st))
    check(lib.spion_linear_backward_weight(ref(td), ref(tx), 1, P(dW.data_ptr()), P(db.data_ptr()), P(ws.data_ptr()), T, K, N, st))
    W, b, dY = torch.cat(Ws).double(), torch.cat(bs).double(), cat(dYs)
    for got, want in ((cat(Ys), X.double() @ W.t() + b), (dX.double(), dY @ W), (dW.double(), dY.t() @ X.double())):
        want = want.float().double()                              # beyond fp32: an infinity
        # within a factor of two of the largest fp32 number the order of the additions decides whether a sum overflows
        sure = ~((want.abs() > 1.7e38) & want.isfinite()) & ~((got.abs() > 1.7e38) & got.isfinite())
        odd = sure & ~want.isfinite()
        assert odd.any() and ((got == want) | (got.isnan() & want.isnan()))[odd].all()
        huge, usual = sure & want.isfinite() & (want.abs() > 1e30), sure & (want.abs() <= 1e30)
        assert ((got - want).abs()[huge] <= 1e-6 * want.abs()[huge]).all()
        assert ((got - want)[usual].norm() <= 2e-6 * want[usual].norm())


@pytest.mark.parametrize("kind,K,N,slices", [("forward", 512, 512, 4), ("forward", 384, 192, 1), ("forward", 768, 96, 1), ("gelu", 640, 96, 1), ("gelu", 768, 384, 4),
                                             ("gradient", 512, 512, 4), ("gradient", 256, 1024, 4), ("gradient_fp32", 512, 256, 2)])
def test_wide_layers_keep_their_columns(kind, K, N, slices):
    """Tables and tiles of the outputs leave wide weights the columns that fit beside a ring alone: A is fetched once per slice of them."""
    import json
    import os
    import tempfile
    T = 149 * 128
    P, st = ctypes.c_void_p, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    one, ref = lambda t: (P * 3)(t.data_ptr(), None, None), ctypes.byref
    X = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16)
    Y = torch.empty(T, N, device="cuda", dtype=torch.float32 if kind == "gradient_fp32" else torch.bfloat16)
    G, W, b = torch.empty(T, N, device="cuda", dtype=torch.bfloat16), torch.zeros(N * K, device="cuda"), torch.zeros(N, device="cuda")

    def call():
        if kind.startswith("gradient"):
            check(lib.spion_linear_backward_input(ref(_tokens([X])), one(W), 1, 0, None, ref(_tokens([Y])), T, N, K, st))
        else:
            check(lib.spion_linear_forward(ref(_tokens([X])), one(W), one(b), 1, 0, ref(_tokens([Y])), P(G.data_ptr()) if kind == "gelu" else None, T, K, N, st))

    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as f:
            grids = [e["args"]["grid"] for e in json.load(f)["traceEvents"] if "k_lin_gemm" in e.get("name", "")]
    assert len(grids) == 1 and grids[0][1] == slices
