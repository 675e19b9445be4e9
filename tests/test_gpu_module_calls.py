"""What callers do with the modules between and around the kernels: several masks before a backward, changed outputs, hooks, transforms
of the framework, copies of modules."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu

B, H, L, D, BS = 2, 2, 256, 32, 64
KINDS = {"native bf16": (True, "bf16"), "native fp32": (True, "fp32"), "drop-in": (False, "fp32")}


def config(native=True, dtype="fp32", task="lra-text", **more):
    return dict({"head_dim": D, "num_head": H, "max_seq_len": L, "batch_size": B, "block_size": BS, "transformer_dim": H * D,
                 "task": task, "native": native, "dtype": dtype}, **more)


def make_layer(kind, dense=False, task="lra-text", seed=0):
    from spion_b200.attention import Attention
    native, dtype = KINDS[kind]
    torch.manual_seed(seed)
    cfg = config(native, dtype, task)
    layer = Attention(cfg).cuda()
    if not dense:
        layer.reconstruct_for_blocksparse(cfg)
    return layer


def amp(kind):
    return torch.autocast("cuda", dtype=torch.bfloat16) if KINDS[kind][1] == "bf16" else contextlib.nullcontext()


def make_mask(seed, density=0.5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mat = (torch.rand(L // BS, L // BS, generator=g, device="cuda") < density).float()
    mat.fill_diagonal_(1)
    return mat


def make_inputs(seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(B, L, H * D, generator=g, device="cuda", requires_grad=True)
    keys = torch.ones(B, L, device="cuda")
    keys[1, L // 2:] = 0
    return x, keys


def run_layer(layer, kind, x, keys, mat):
    with amp(kind):
        return layer(x, keys, mat)[0]


def gradients(layer, out, x):
    return torch.autograd.grad(out.float().square().sum(), [x] + list(layer.parameters()))


def same(a, b):
    assert len(a) == len(b)
    for s, t in zip(a, b):
        assert torch.equal(s, t), float((s - t).abs().max())


def test_two_masks_before_the_backward_of_a_drop_in_layer():
    """Every call's backward runs on the mask of its own forward, whatever the layer was called with since."""
    kind, masks = "drop-in", (make_mask(1, 0.2), make_mask(2, 0.9))
    x, keys = make_inputs()
    want = []
    for mat in masks:
        layer = make_layer(kind)
        want.append(gradients(layer, run_layer(layer, kind, x, keys, mat), x))
    layer = make_layer(kind)
    outs = [run_layer(layer, kind, x, keys, mat) for mat in masks]
    for i in (0, 1):
        same(gradients(layer, outs[i], x), want[i])


@pytest.mark.parametrize("bs", [64, 32])
@pytest.mark.parametrize("dtype,recompute", [(torch.bfloat16, True), (torch.bfloat16, False), (torch.float32, None)])
def test_two_masks_before_the_backward_of_a_native_module(dtype, recompute, bs):
    from spion_b200.native import BlockSparseAttention
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B, H, L, D, generator=g, device="cuda").to(dtype).requires_grad_() for _ in range(3))
    masks = [(torch.rand(L // bs, L // bs, generator=g, device="cuda") < p).float() + torch.eye(L // bs, device="cuda") for p in (0.2, 0.8)]

    def module():
        return BlockSparseAttention(dict(config(), block_size=bs), dtype=dtype, recompute=recompute)

    def grads(out):
        return torch.autograd.grad(out.float().square().sum(), (q, k, v))

    want = [grads(module()(q, k, v, None, mat)[0]) for mat in masks]
    mod = module()
    outs = [mod(q, k, v, None, mat)[0] for mat in masks]
    same(grads(outs[0]), want[0])
    assert torch.equal(mod(q, k, v)[0], outs[1])                 # the module is on its last mask again
    same(grads(outs[1]), want[1])


@pytest.mark.parametrize("dtype,recompute", [(torch.bfloat16, True), (torch.bfloat16, False), (torch.float32, None)])
@pytest.mark.parametrize("what", ["output", "probabilities"])
def test_a_changed_output_is_noticed(dtype, recompute, what):
    """The backward reads the output (and, where they are stored, the probabilities): a change in between is an error."""
    from spion_b200.native import BlockSparseAttention
    if what == "probabilities" and recompute:
        pytest.skip("the rebuilt path does not read them")
    q, k, v = (torch.randn(B, H, L, D, device="cuda").to(dtype).requires_grad_() for _ in range(3))
    mod = BlockSparseAttention(config(), dtype=dtype, recompute=recompute)
    out, probs = mod(q, k, v, None, make_mask(4))
    total = out.float().sum()
    if what == "output":
        out.mul_(2.0)
        total = out.float().sum()
    else:
        probs.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        total.backward()


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("padded", [False, True])
def test_gradients_of_a_call_that_returns_its_probabilities(d, padded):
    """Blocks of 64: the backward reads the P that the caller got, so the gradients are those of the stored path bit for bit and a
    change of P in between is an error."""
    from spion_b200.native import BlockSparseAttention
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k, v, do = (torch.randn(B, H, L, d, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_()
    keys = make_inputs()[1]
    got = []
    for recompute in (None, False):
        mod = BlockSparseAttention(config(head_dim=d, transformer_dim=H * d), dtype=torch.bfloat16, keypad=padded, recompute=recompute)
        out, probs = mod(q, k, v, keys, make_mask(4))
        got.append((out, probs) + torch.autograd.grad(out, (q, k, v), do))
    same(*got)
    mod = BlockSparseAttention(config(head_dim=d, transformer_dim=H * d), dtype=torch.bfloat16, keypad=padded)
    out, probs = mod(q, k, v, keys, make_mask(4))
    probs.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(do)


@pytest.mark.parametrize("d,batch", [(32, 2), (32, 1023), (32, 1024), (64, 2)])
def test_one_backward_path_for_a_layer_and_a_direct_call(d, batch):
    """The path follows from the problem and not from the module that asks (16 selected blocks: 2 * 1024 * 16 is the bound at 32)."""
    from spion_b200.attention import Attention
    from spion_b200.native import BlockSparseAttention
    cfg = config(dtype="bf16", head_dim=d, transformer_dim=H * d, batch_size=batch, max_seq_len=512)
    mat = torch.eye(8, device="cuda") + torch.diag(torch.ones(7, device="cuda"), 1)
    mat[7, 0] = 1
    layer = Attention(cfg).cuda()
    layer.reconstruct_for_blocksparse(cfg)
    mod = BlockSparseAttention(cfg, dtype=torch.bfloat16, keypad=True, return_probs=False)
    for m in (layer.block_attn, mod):
        m.set_mask(mat)
    assert mod.nnzb == 16 and mod.recompute == layer.block_attn.recompute == (d == 64 or batch == 1024)
    g = torch.Generator(device="cuda").manual_seed(8)
    q, k, v, do = (torch.randn(batch, H, 512, d, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_()
    keys = torch.ones(batch, 512, device="cuda")
    same(*(torch.autograd.grad(m(q, k, v, keys)[0], (q, k, v), do) for m in (layer.block_attn, mod)))


def test_changed_probabilities_of_a_drop_in_layer_are_noticed():
    layer, (x, keys) = make_layer("drop-in", task="lra-image"), make_inputs()
    out, probs = layer(x, keys, make_mask(4))
    probs.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


@pytest.mark.parametrize("kind", list(KINDS))
def test_hooks_on_saved_tensors_see_all_of_them(kind):
    """Saved tensors may be packed elsewhere, in other strides, and rebuilt: same gradients."""
    from torch.utils.checkpoint import checkpoint
    x, keys = make_inputs()
    layer, mat = make_layer(kind), make_mask(5)
    xb = x.detach().to(torch.bfloat16).requires_grad_() if KINDS[kind][1] == "bf16" else x
    for inp in (x, xb):                                          # bf16 input: operands in the other layout
        want = gradients(layer, run_layer(layer, kind, inp, keys, mat), inp)
        sizes = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (sizes.append(t.numel()), t.cpu().contiguous())[1], lambda t: t.cuda()):
            out = run_layer(layer, kind, inp, keys, mat)
        same(gradients(layer, out, inp), want)
        assert sum(sizes) >= 5 * B * L * H * D                   # input, Q, K, V, O
        again = checkpoint(lambda t: run_layer(layer, kind, t, keys, mat), inp, use_reentrant=False)
        same(gradients(layer, again, inp), want)


@pytest.mark.parametrize("kind", list(KINDS))
def test_a_failing_backward_raises_the_library_s_error(kind):
    from spion_b200._lib import SpionError
    x, keys = make_inputs()
    layer, mat = make_layer(kind), make_mask(6)
    out = run_layer(layer, kind, x, keys, mat)
    block = layer.block_attn
    ctx = block._ctx if KINDS[kind][0] else block.context(mat)
    handle, ctx.handle = ctx.handle, 0                            # every call of the library refuses it
    try:
        with pytest.raises(SpionError, match="failed"):
            out.sum().backward()
    finally:
        ctx.handle = handle


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("kind", list(KINDS))
def test_transforms_of_the_framework(kind, dense):
    """Tracing records the call; forward-mode tangents, which nothing here forms, are refused and not dropped."""
    import torch.autograd.forward_ad as fw
    x, keys = make_inputs()
    layer, mat = make_layer(kind, dense), None if dense else make_mask(7)

    class Call(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.layer = layer

        def forward(self, t):
            return run_layer(layer, kind, t, keys, mat)

    call = Call()
    with torch.no_grad():
        traced = torch.jit.trace(call, (x,), check_trace=False)
        other = torch.randn_like(x)
        got, want = traced(other).float(), call(other).float()
    # stage by stage instead of one node: other roundings of the same products
    assert float((got - want).norm() / want.norm()) < (2e-2 if KINDS[kind][1] == "bf16" else 1e-5)
    with fw.dual_level(), pytest.raises(NotImplementedError):
        call(fw.make_dual(x.detach(), torch.ones_like(x)))
    assert not torch.isnan(call(x)).any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_transforms_of_an_attention_call(dtype):
    import torch.autograd.forward_ad as fw
    from spion_b200.native import BlockSparseAttention
    q, k, v = (torch.randn(B, H, L, D, device="cuda").to(dtype).requires_grad_() for _ in range(3))
    mod = BlockSparseAttention(config(), dtype=dtype)
    mod.set_mask(make_mask(8))
    call = lambda *t: mod(*t)[0]
    traced = torch.jit.trace(call, (q, k, v), check_trace=False)
    other = torch.randn_like(q).requires_grad_()
    got, want = (torch.autograd.grad(f(other, k, v).float().square().sum(), (other, k, v)) for f in (traced, call))
    same(got, want)
    with fw.dual_level(), pytest.raises(NotImplementedError):
        call(fw.make_dual(q.detach(), torch.ones_like(q)), k, v)


def test_transforms_of_a_linear_layer():
    import torch.autograd.forward_ad as fw
    from torch.fx.experimental.proxy_tensor import make_fx
    from spion_b200.layernorm import BiasGradLinear
    lin, x, other = BiasGradLinear(64, 128).cuda(), torch.randn(50, 64, device="cuda"), torch.randn(50, 64, device="cuda")
    want = lin(other)
    for f in (torch.jit.trace(lin, (x,), check_trace=False), make_fx(lambda t: lin(t))(x)):
        assert float((f(other) - want).norm() / want.norm()) < 1e-5
    with fw.dual_level(), pytest.raises(NotImplementedError):
        lin(fw.make_dual(x, torch.ones_like(x)))
    with pytest.raises(RuntimeError):
        torch.func.vmap(lin)(x[None].expand(3, -1, -1))


def second_order(layer, kind, x, keys, mat):
    out = run_layer(layer, kind, x, keys, mat)
    first = torch.autograd.grad(out.float().square().sum(), [x] + list(layer.parameters()), create_graph=True)
    total = sum(g.float().square().sum() for g in first if g.requires_grad)
    second = torch.autograd.grad(total, [x] + list(layer.parameters()), allow_unused=True) if torch.is_tensor(total) else ()
    return first, second


@pytest.mark.parametrize("kind", list(KINDS))
def test_a_recorded_backward_of_a_layer(kind):
    """create_graph: the same first gradients, and the second ones that the stages one by one give."""
    x, keys = make_inputs()
    layer, mat = make_layer(kind), make_mask(9)
    if KINDS[kind][1] == "bf16":
        x = x.detach().to(torch.bfloat16).requires_grad_()
    plain = gradients(layer, run_layer(layer, kind, x, keys, mat), x)
    first, second = second_order(layer, kind, x, keys, mat)
    hook = layer.W_k.register_forward_hook(lambda *_: None)       # stage by stage
    want_first, want_second = second_order(layer, kind, x, keys, mat)
    hook.remove()
    tol = 3e-2 if KINDS[kind][1] == "bf16" else 1e-5              # bf16: a chain of roundings of 2^-9 in another order
    close = lambda a, b: float((a.float() - b.float()).norm()) <= tol * float(b.float().norm()) + 1e-6
    assert all(close(a.detach(), b) for a, b in zip(first, plain))
    assert all(close(a.detach(), b.detach()) for a, b in zip(first, want_first))
    assert [g is None for g in second] == [g is None for g in want_second]
    assert all(close(a, b) for a, b in zip(second, want_second) if a is not None)


def test_second_derivatives_of_linear_layers():
    from spion_b200._ops import ops
    from spion_b200.layernorm import BiasGradLinear
    lin, l2 = BiasGradLinear(64, 128).cuda(), torch.nn.Linear(128, 64).cuda()
    x = torch.randn(50, 64, device="cuda", requires_grad=True)

    def penalty(f, x, params):
        g = torch.autograd.grad(f(x).square().sum(), x, create_graph=True)[0]
        return torch.autograd.grad(g.square().sum(), [x] + params)

    got = penalty(lin, x, [lin.weight])
    w, xd = lin.weight.detach().double().requires_grad_(), x.detach().double().requires_grad_()
    want = penalty(lambda t: torch.nn.functional.linear(t, w, lin.bias.detach().double()), xd, [w])
    assert all(float((a - b).norm() / b.norm()) < 1e-6 for a, b in zip(got, want))
    # mixed precision: through the input
    xb = x.detach().to(torch.bfloat16).requires_grad_()
    ff = lambda t: ops.mlp(t, lin.weight, lin.bias, l2.weight, l2.bias)
    got = penalty(ff, xb, [])
    ref = lambda t: torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(t, w, lin.bias.double())), l2.weight.double(), l2.bias.double())
    want = penalty(ref, xb.detach().double().requires_grad_(), [])
    assert float((got[0].double() - want[0]).norm() / want[0].norm()) < 3e-2


@pytest.mark.parametrize("what", ["input", "weights"])
@pytest.mark.parametrize("call", ["layer", "linear", "feed-forward"])
def test_mixed_precision_calls_keep_what_their_backward_reads(call, what):
    """Under autocast the casts are copies: the fp32 input and the weights may change before the backward, as with torch.nn.Linear."""
    from spion_b200._ops import ops
    from spion_b200.layernorm import BiasGradLinear
    x, keys = make_inputs()
    if call == "layer":
        mod, mat = make_layer("native bf16"), make_mask(10)
        f = lambda t: mod(t, keys, mat)[0]
    elif call == "linear":
        mod = BiasGradLinear(H * D, 96).cuda()
        f = mod
    else:
        mod = torch.nn.Sequential(BiasGradLinear(H * D, 160), BiasGradLinear(160, H * D)).cuda()
        f = lambda t: ops.mlp(t, mod[0].weight, mod[0].bias, mod[1].weight, mod[1].bias)
    params = list(mod.parameters())

    def grads(change):
        h = x * 1.0
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = f(h)
        old = [p.detach().clone() for p in params]
        if change:
            with torch.no_grad():
                if what == "input":
                    h.mul_(3.0)
                else:
                    for p in params:
                        p.mul_(3.0)
        g = torch.autograd.grad(y.float().square().sum(), [x] + params)
        with torch.no_grad():
            for p, o in zip(params, old):
                p.copy_(o)
        return g

    same(grads(True), grads(False))


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("kind", list(KINDS))
def test_hooks_and_replacements_of_the_attention_module(kind, dense):
    """What is hooked into or put in the place of the attention module of a layer is called."""
    x, keys = make_inputs()
    layer, mat = make_layer(kind, dense), None if dense else make_mask(11)
    want = run_layer(layer, kind, x, keys, mat)
    name = "attn" if dense else "block_attn"
    inner = getattr(layer, name)
    calls = []
    hook = inner.register_forward_hook(lambda *_: calls.append("hook"))
    got = run_layer(layer, kind, x, keys, mat)
    hook.remove()
    assert calls == ["hook"]
    tol = 2e-2 if KINDS[kind][1] == "bf16" else 1e-5              # stage by stage: other roundings of the same products
    assert float((got.float() - want.float()).norm()) <= tol * float(want.float().norm())
    everywhere = torch.nn.modules.module.register_module_forward_hook(lambda m, *_: calls.append(type(m).__name__))
    run_layer(layer, kind, x, keys, mat)
    everywhere.remove()
    assert {type(layer).__name__, type(inner).__name__, type(layer.W_q).__name__} <= set(calls)

    class Other(torch.nn.Module):
        def forward(self, q, k, v, *rest):
            calls.append("other")
            return inner(q, k, v, *rest)

    setattr(layer, name, Other())
    run_layer(layer, kind, x, keys, mat)
    assert calls[-1] == "other"
    setattr(layer, name, inner)
    assert torch.equal(run_layer(layer, kind, x, keys, mat), want)


@pytest.mark.parametrize("what", ["hook", "activation", "approximate", "second layer in bf16", "no bias", "dropout of its own"])
def test_the_fused_feed_forward_serves_the_block_as_it_was_made(what):
    """Anything hooked, replaced or switched on in the block runs; the reference is the block called as the module it is."""
    from spion_b200 import harness
    cfg = harness.task_config("text", B, dtype="bf16")
    cfg.update(max_seq_len=L, dropout_prob=0.0)
    torch.manual_seed(0)
    layer = harness.TransformerLayer(cfg).cuda()
    block, x, calls = layer.mlpblock, torch.randn(B, L, 64, device="cuda"), []
    if what == "hook":
        for m in block:
            m.register_forward_hook(lambda m, *_: calls.append(type(m).__name__))
    elif what == "activation":
        block[1] = torch.nn.ReLU()
    elif what == "approximate":
        block[1] = torch.nn.GELU(approximate="tanh")
    elif what == "second layer in bf16":
        block[3].to(torch.bfloat16)
    elif what == "no bias":
        block[3].bias = None
    else:
        layer.eval()
        block[2].p = 1.0
        block[2].train()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        got, want = layer.feed_forward(x), block(x)
    assert torch.equal(got, want)
    if what == "hook":
        assert calls[:5] == ["BiasGradLinear", "GELU", "Dropout", "BiasGradLinear", "Dropout"]
    if what == "dropout of its own":
        assert torch.equal(got, block[3].bias.to(got.dtype).expand_as(got))


def test_the_fused_feed_forward_saves_all_it_reads():
    from spion_b200 import harness
    cfg = harness.task_config("text", B, dtype="bf16")
    cfg.update(max_seq_len=L, dropout_prob=0.0)
    layer = harness.TransformerLayer(cfg).cuda()
    x = torch.randn(B, L, 64, device="cuda", requires_grad=True)
    grads = lambda y: torch.autograd.grad(y.float().square().sum(), [x] + list(layer.mlpblock.parameters()))
    sizes = []
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = grads(layer.feed_forward(x))
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (sizes.append(t.numel()), t.cpu())[1], lambda t: t.cuda()):
            y = layer.feed_forward(x)
    same(grads(y), want)
    assert sum(sizes) >= B * L * (64 + 2 * 128)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("kind", list(KINDS))
def test_key_padding_masks_of_one_sequence(kind, dense):
    """The drop-in layers broadcast them; the native ones refuse them."""
    from spion_b200._lib import SpionError
    x, keys = make_inputs()
    layer, mat = make_layer(kind, dense), None if dense else make_mask(12)
    for small in (keys[1:], keys[:, :1]):
        if KINDS[kind][0]:
            with pytest.raises(SpionError, match="key-padding mask"):
                run_layer(layer, kind, x, small, mat)
        else:
            assert torch.equal(run_layer(layer, kind, x, small, mat), run_layer(layer, kind, x, small.expand(B, L).contiguous(), mat))


@pytest.mark.parametrize("dense", [False, True])
def test_a_drop_in_layer_can_be_copied(dense):
    """copy.deepcopy, as averaged models do: the copy shares the attention library's handle and has weights of its own."""
    import copy
    kind = "drop-in"
    x, keys = make_inputs()
    layer, mat = make_layer(kind, dense), None if dense else make_mask(13)
    other = copy.deepcopy(layer)
    want = run_layer(layer, kind, x, keys, mat)
    assert torch.equal(run_layer(other, kind, x, keys, mat), want)
    with torch.no_grad():
        other.W_v.weight.zero_()
    assert torch.equal(run_layer(layer, kind, x, keys, mat), want)


@pytest.mark.parametrize("kind", list(KINDS))
def test_masks_that_share_an_address(kind):
    """A mask and its transpose, and a mask tensor that has been given other storage, are different masks."""
    x, keys = make_inputs()
    mat = make_mask(14, 0.4)
    mat[0, 3], mat[3, 0] = 1, 0
    fresh = lambda m: run_layer(make_layer(kind), kind, x, keys, m.clone())
    layer = make_layer(kind)
    assert torch.equal(run_layer(layer, kind, x, keys, mat), fresh(mat))
    assert torch.equal(run_layer(layer, kind, x, keys, mat.t()), fresh(mat.t()))
    run_layer(layer, kind, x, keys, mat)
    mat.data = make_mask(15, 0.9)
    assert torch.equal(run_layer(layer, kind, x, keys, mat), fresh(mat))


def test_a_wait_of_a_linear_layer_that_gave_up_is_reported():
    """By the check of the attention module in the same layer; until then the linear kernels leave at once."""
    from spion_b200._lib import SpionError, check, lib
    from spion_b200.layernorm import BiasGradLinear
    kind = "native bf16"
    x, keys = make_inputs()
    layer, mat, lin = make_layer(kind), make_mask(16), BiasGradLinear(64, 64).cuda()
    want, want_lin = run_layer(layer, kind, x, keys, mat), lin(x)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()                             # a non-blocking stream: no order with the legacy one
    with torch.cuda.stream(stream):
        check(lib.spion_linear_selftest_bounded_wait(1000, stream.cuda_stream))
        assert lib.spion_linear_status(0) != 0
        grads = torch.autograd.grad(lin(x).sum(), list(lin.parameters()))      # returns, whatever it left in its buffers
        del grads
    torch.cuda.synchronize()
    with pytest.raises(SpionError, match="timed out"):
        layer.block_attn.check_device_status()
    layer.block_attn.check_device_status()
    assert lib.spion_linear_status(0) == 0
    assert torch.equal(lin(x), want_lin) and torch.equal(run_layer(layer, kind, x, keys, mat), want)


def test_modules_of_several_threads():
    """Modules made and called by several threads at once give what they give one after another."""
    import threading
    x, keys = make_inputs()
    kinds = list(KINDS) * 2
    masks = [make_mask(20 + i) for i in range(len(kinds))]
    got, failed = [None] * len(kinds), []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                layer = layers[i]
                if not KINDS[kinds[i]][0] or KINDS[kinds[i]][1] == "fp32":
                    layer = make_copy(layer, kinds[i])
                for _ in range(3):
                    out = run_layer(layer, kinds[i], x, keys, masks[i])
                    g = gradients(layer, out, x)
                got[i] = [out.detach(), *g]
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            failed.append(e)

    def make_copy(layer, kind):                                  # torch's seed is the process's: the weights come from outside
        native, dtype = KINDS[kind]
        from spion_b200.attention import Attention
        cfg = config(native, dtype)
        other = Attention(cfg).cuda()
        other.load_state_dict(layer.state_dict())
        other.reconstruct_for_blocksparse(cfg)
        return other

    layers = [make_layer(k) for k in kinds]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(kinds))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for i, kind in enumerate(kinds):
        layer = make_layer(kind)
        out = run_layer(layer, kind, x, keys, masks[i])
        same(got[i], [out.detach(), *gradients(layer, out, x)])


def test_memory_of_contexts():
    """With more in use than the pool keeps, what one context gives back is there for the next; in the end all but that goes back."""
    from spion_b200.native import BlockSparseAttention

    def context(heads):                                          # 2 * 4 bytes of workspace per row and matrix
        mod = BlockSparseAttention(dict(config(), num_head=heads, max_seq_len=4096), dtype=torch.bfloat16)
        mod.set_mask(torch.eye(64, device="cuda"))
        return mod

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    context(1)
    torch.cuda.empty_cache()
    start = free()
    large, small = context(2048), context(256)                   # 134 MB and 17 MB
    both = free()
    assert start - both > 100 << 20
    del small
    assert free() == both
    small = context(256)
    assert free() == both
    del large, small
    assert start - free() < 80 << 20
