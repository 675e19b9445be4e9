"""Performance cases of the block-sparse attention framework, measured through its public entry points.

What a user of the framework has it do, from the smallest call to the largest:

* ``attn``     one ``native.BlockSparseAttention`` call: forward alone (``grad`` False) or forward + backward, the
               kernel-sweep form (Q, K, V ~ N(0,1), mask = two-block diagonal band + random blocks);
* ``layer``    one multi-head ``attention.Attention`` layer (projections, attention, output projection) as an encoder calls
               it: the sparse phase of training, the dense warm-up phase with the mean attention map that pattern discovery
               reads, or inference; on the native path (``native`` True) or behind the reference's own entry points;
* ``pattern``  pattern discovery of the layers of a model from their mean attention maps;
* ``train``    one captured optimizer step of the encoder classifier (``harness.Trainer``).

Tasks with padded inputs (text, retrieval) carry a key-padding mask with a ragged tail per sequence.
"""
import math
from contextlib import nullcontext

import numpy as np
import torch

from spion_b200 import harness, pattern, synthetic
from spion_b200.attention import Attention
from spion_b200.native import BlockSparseAttention

DEVICE = "cuda"
TASKS = {False: "lra-image", True: "lra-text"}          # without / with key padding


def _attn(name, B, H, L, d, bs, density, dtype, grad=True, probs=False, keypad=False, stripes=0):
    return {"name": name, "kind": "attn", "B": B, "H": H, "L": L, "d": d, "bs": bs, "density": density, "dtype": dtype,
            "grad": grad, "probs": probs, "keypad": keypad, "stripes": stripes}


def _layer(name, B, H, L, d, bs, density, dtype, native=True, phase="sparse", grad=True, keypad=False, stripes=0):
    return {"name": name, "kind": "layer", "B": B, "H": H, "L": L, "d": d, "bs": bs, "density": density, "dtype": dtype,
            "native": native, "phase": phase, "grad": grad, "keypad": keypad, "stripes": stripes}


def _pattern(name, L, bs, layers, q):
    return {"name": name, "kind": "pattern", "L": L, "bs": bs, "layers": layers, "q": q}


def _train(name, task, B, L, dtype, q):
    return {"name": name, "kind": "train", "task": task, "B": B, "L": L, "dtype": dtype, "q": q}


def listed():
    return [
        # classifying a single sequence with a trained model: latency and launches are everything
        _layer("infer_one_sequence", 1, 2, 1024, 32, 64, 0.12, "bf16", grad=False, keypad=True),
        # one attention layer of the image-shaped encoder at a small batch, fp32, forward + backward
        _attn("layer_fp32_small", 8, 2, 1024, 32, 32, 0.15, "fp32"),
        # kernel sweep at L = 4096, blocks of 64, with the probabilities handed back (the module's default)
        _attn("sweep_L4096_bs64", 8, 8, 4096, 64, 64, 0.05, "bf16", probs=True),
        # the same with blocks of 32
        _attn("sweep_L4096_bs32", 8, 8, 4096, 64, 32, 0.05, "bf16"),
        # long sequences, the largest call of the sweep
        _attn("long_L16384_bs64", 8, 8, 16384, 64, 64, 0.05, "bf16"),
        # attention layer of the retrieval-shaped dual encoder at 64 pairs: mixed precision, padded keys, a few
        # block columns that every row attends to (as discovered masks have)
        _layer("retrieval_layer_bf16", 128, 2, 4096, 32, 64, 0.10, "bf16", keypad=True, stripes=2),
        # attention layer of the image-shaped encoder at the training batch, fp32
        _layer("image_layer_fp32", 256, 2, 1024, 32, 32, 0.15, "fp32"),
        # sparse phase behind the reference's entry points (fp32, element-CSR probabilities), odd sizes, padded keys
        _layer("dropin_sparse_odd", 5, 3, 3008, 64, 64, 0.08, "fp32", native=False, keypad=True, stripes=1),
        # dense warm-up phase behind the reference's entry points, with the mean attention map
        _layer("dropin_dense_warmup", 8, 2, 1024, 32, 32, 1.0, "fp32", native=False, phase="dense"),
        # dense warm-up phase on the native path, odd sizes, padded keys
        _layer("native_dense_warmup_odd", 9, 2, 1984, 32, 64, 1.0, "bf16", phase="dense", keypad=True),
        # the dense -> sparse switch: block masks of a two-layer model from its mean attention maps
        _pattern("discover_L4096", 4096, 64, 2, 0.96),
        # optimizer step of the retrieval-shaped dual encoder at the per-GPU share of an eight-GPU run
        _train("train_retrieval_8_pairs", "retrieval", 8, 4096, "bf16", 0.90),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["attn"] * 4 + ["sparse"] * 4 + ["dense"] * 2 + ["pattern", "train"])
    bs = rng.choice([32, 64])
    d = rng.choice([32, 64])
    if kind == "pattern":
        return _pattern("", _log_int(rng, 512 // bs, 4096 // bs) * bs, bs, rng.choice([1, 2]), rng.choice([0.8, 0.9, 0.96, 0.99]))
    if kind == "train":
        task = rng.choice(["image", "text", "retrieval"])
        B = {"image": _log_int(rng, 4, 48), "text": _log_int(rng, 1, 16), "retrieval": _log_int(rng, 1, 8)}[task]
        L = 1024 if task == "image" else rng.choice([1024, 2048, 4096])
        return _train("", task, B, L, "fp32" if task == "image" else "bf16", rng.choice([0.8, 0.9, 0.95]))
    dtype = rng.choice(["bf16", "bf16", "fp32"])
    keypad = rng.random() < 0.5
    if kind == "dense":
        native = rng.random() < 0.5
        nb = _log_int(rng, 256 // bs, (3072 if native else 1536) // bs)
        nb += nb % 2 if dtype == "bf16" and native and bs == 32 else 0
        H = rng.choice([1, 2, 2, 4])
        return _layer("", _log_int(rng, 1, 32), H, nb * bs, d, bs, 1.0, dtype if native else "fp32", native=native,
                      phase="dense", keypad=keypad)
    top = 16384 if dtype == "bf16" and kind == "attn" else 8192
    nb = _log_int(rng, 256 // bs, top // bs)
    if dtype == "bf16" and bs == 32:
        nb += nb % 2
    density = round(math.exp(rng.uniform(math.log(0.02), math.log(0.30))), 3)
    stripes = rng.choice([0, 0, 1, 2])
    grad = rng.random() < 0.75
    if kind == "attn":
        return _attn("", _log_int(rng, 1, 16), rng.choice([1, 2, 3, 4, 8]), nb * bs, d, bs, density, dtype, grad=grad,
                     probs=rng.random() < 0.4, keypad=keypad, stripes=stripes)
    return _layer("", _log_int(rng, 1, 256), rng.choice([1, 2, 2, 3, 4]), nb * bs, d, bs, density, dtype,
                  native=dtype == "bf16" or rng.random() < 0.5, grad=grad, keypad=keypad, stripes=stripes)


def _cost(case):
    """Rough seconds of a pass, to keep drawn cases within the largest listed one."""
    w = work(case)
    rate = 25e12 if case.get("dtype", "fp32") == "fp32" and case["kind"] != "pattern" else 200e12
    return w["flops"] / rate + w["bytes"] / 2.5e12


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw_once(rng)
        if _cost(c) <= most and (c["kind"] in ("pattern", "train") or _nnzb(c) * c["bs"] ** 2 * c["B"] * c["H"] < 6e8):
            c.pop("name")
            return c


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _nnzb(case):
    nb = case["L"] // case["bs"]
    least = 2 * nb - 1 + case["stripes"] * nb
    return nb * nb if case["density"] >= 1.0 else min(nb * nb, max(int(round(case["density"] * nb * nb)), least))


def _block_mask(seed, case):
    """Diagonal band of two blocks, ``stripes`` full block columns, uniformly random blocks up to the density."""
    nb = case["L"] // case["bs"]
    mat = synthetic.band_random_mask(seed, nb, 0.0)
    rng = np.random.default_rng(seed + 1)
    mat[:, rng.choice(nb, size=min(nb, case["stripes"]), replace=False)] = 1
    extra = _nnzb(case) - int(mat.sum())
    if extra > 0:
        free = np.flatnonzero(mat.ravel() == 0)
        mat.ravel()[rng.choice(free, size=min(extra, free.size), replace=False)] = 1
    return torch.from_numpy(mat.astype(np.float32)).to(DEVICE)


def _attention_map(g, L):
    """Row-stochastic map with a diagonal band, off-diagonal bands and vertical stripes over noise: the shapes of
    trained attention maps (``synthetic.structured_map``, formed on the GPU)."""
    S = torch.randn(L, L, generator=g, device=DEVICE) * 0.5
    i = torch.arange(L, device=DEVICE)
    diff = (i[:, None] - i[None, :]).float()
    S += 4.0 * torch.exp(-((diff / 6.0) ** 2))
    for o in torch.randint(-L // 2, L // 2, (3,), generator=g, device=DEVICE).tolist():
        S += 3.0 * torch.exp(-(((diff - o) / 4.0) ** 2))
    for c in torch.randint(0, L, (4,), generator=g, device=DEVICE).tolist():
        S += (2.5 * torch.exp(-(((i - c).float() / 3.0) ** 2)))[None, :]
    return torch.softmax(S, dim=-1).contiguous()


def _config(case, **more):
    H, d = case["H"], case["d"]
    return dict({"head_dim": d, "num_head": H, "max_seq_len": case["L"], "batch_size": case["B"], "block_size": case["bs"],
                 "transformer_dim": H * d, "task": TASKS[case["keypad"]], "dtype": case["dtype"]}, **more)


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "pattern":
        return {"case": case, "maps": [_attention_map(g, case["L"]) for _ in range(case["layers"])],
                "config": {"block_size": case["bs"], "max_seq_len": case["L"], "threshold": case["q"]}}
    if kind == "train":
        return _prepare_train(case, seed, g)
    B, H, L, d = case["B"], case["H"], case["L"], case["d"]
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    mask = synthetic.key_padding(seed, B, L).to(DEVICE) if case["keypad"] else torch.ones(B, L, device=DEVICE)
    state = {"case": case, "mask": mask, "mat": _block_mask(seed, case)}
    if kind == "attn":
        q, k, v, do = (torch.randn(B, H, L, d, generator=g, device=DEVICE).to(dtype) for _ in range(4))
        for t in (q, k, v):
            t.requires_grad_(case["grad"])
        mod = BlockSparseAttention(_config(case), dtype=dtype, keypad=case["keypad"], return_probs=case["probs"])
        mod.set_mask(state["mat"])
        state.update(mod=mod, qkv=(q, k, v), do=do)
        return state
    torch.manual_seed(seed)
    config = _config(case, native=case["native"])
    layer = Attention(config, inference=not case["grad"]).to(DEVICE)
    if case["phase"] == "sparse":
        layer.reconstruct_for_blocksparse(config)
    layer.train(case["grad"])
    x = torch.randn(B, L, H * d, generator=g, device=DEVICE)
    x.requires_grad_(case["grad"])
    do = torch.randn(B, L, H * d, generator=g, device=DEVICE).to(dtype)
    state.update(layer=layer, x=x, do=do, params=list(layer.parameters()))
    return state


def _prepare_train(case, seed, g):
    # dropout is the framework user's regulariser and draws fresh random numbers; off, so that outputs can be compared
    cfg = harness.task_config(case["task"], case["B"], native=True, dtype=case["dtype"])
    cfg.update(max_seq_len=case["L"], dropout_prob=0.0, attention_dropout=0.0, threshold=case["q"])
    trainer = harness.Trainer(cfg, lr=1e-4, device=torch.device(DEVICE, torch.cuda.current_device()), seed=seed)
    trainer.discover([_attention_map(g, case["L"]) for _ in range(cfg["num_layers"])])
    B, L = case["B"], case["L"]

    def ids():
        t = torch.randint(1, cfg["vocab_size"], (B, L), generator=g, device=DEVICE)
        if case["task"] != "image":                                   # padded tail, as the text tasks have
            keep = torch.randint(L // 2, L + 1, (B, 1), generator=g, device=DEVICE)
            t = torch.where(torch.arange(L, device=DEVICE)[None, :] < keep, t, 0)
        return t

    x = (ids(), ids()) if cfg["dual"] else ids()
    y = torch.randint(0, cfg["num_classes"], (B,), generator=g, device=DEVICE)
    trainer.capture_sparse_step(x, y)
    return {"case": case, "trainer": trainer, "ids": x, "labels": y,
            "weights": [p for p in trainer.model.parameters() if p.dim() > 1]}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pattern":
        mats, patterns = pattern.discover_layers(state["maps"], state["config"])
        # the index arrays of the block structure have a length of their own for every map; they follow from ``mat``
        return {"mats": mats, "patterns": [[p.nnzb, p.mat, p.pooled, p.thresh, p.row_ptr, p.col_ptr] for p in patterns]}
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.step_graph(state["ids"], state["labels"])
        return {"loss": loss, "grads": trainer.bucket.flat, "weights": state["weights"]}
    if kind == "attn":
        return _run_attn(state, case)
    return _run_layer(state, case)


def _run_attn(state, case):
    q, k, v = state["qkv"]
    if not case["grad"]:
        with torch.no_grad():
            out, probs = state["mod"](q, k, v, state["mask"])
        return {"out": out, "probs": probs if case["probs"] else None}
    out, probs = state["mod"](q, k, v, state["mask"])
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["do"])
    return {"out": out, "probs": probs if case["probs"] else None, "dq": dq, "dk": dk, "dv": dv}


def _run_layer(state, case):
    layer, x, mask = state["layer"], state["x"], state["mask"]
    amp = torch.autocast("cuda", dtype=torch.bfloat16) if case["dtype"] == "bf16" else nullcontext()
    mat = state["mat"] if case["phase"] == "sparse" else None
    if not case["grad"]:
        with torch.no_grad(), amp:
            out, _ = layer(x, mask, mat)
        return {"out": out}
    result = {}
    with amp:
        out, attn = layer(x, mask, mat)
    if mat is None and case["native"]:
        result["map"] = layer.attn.mean_attention_map(attn)
    elif mat is None:
        result["map"] = pattern.mean_attention_map(attn.permute(0, 1, 3, 2), transposed_storage=True)
        result["attn"] = attn
    elif not case["native"] and not case["keypad"]:
        result["attn"] = attn
    result["out"] = out
    result["grads"] = torch.autograd.grad(out, [x] + state["params"], state["do"])
    return result


# ------------------------------------------------------------------------------------------------ measures
def work(case):
    kind = case["kind"]
    if kind == "pattern":
        return {"bytes": 4.0 * case["L"] ** 2 * case["layers"], "flops": 4.0 * case["L"] ** 2 * case["layers"]}
    if kind == "train":
        return _work_train(case)
    B, H, L, d = case["B"], case["H"], case["L"], case["d"]
    e = 2 if case["dtype"] == "bf16" else 4
    values = float(_nnzb(case)) * case["bs"] ** 2 * B * H
    operand = float(B) * H * L * d
    # attention: S and O forward, dP, dQ, dK, dV backward; Q, K, V in, O out, then Q, K, V, O, dO in, dQ, dK, dV out
    flops = (12.0 if case["grad"] else 4.0) * values * d
    size = (12 if case["grad"] else 4) * operand * e
    if kind == "attn":
        return {"flops": flops, "bytes": size + (values * e if case["probs"] else 0)}
    # layer: x in, out out; upstream gradient in, dx out; four projections of width H * d
    dim = float(H * d)
    flops += 8.0 * B * L * dim * dim * (3 if case["grad"] else 1)
    size += B * L * dim * (4 + e + ((e + 4) if case["grad"] else 0))
    if case["phase"] == "dense":
        size += 4.0 * L * L
    if not case["native"] and (case["phase"] == "dense" or not case["keypad"]):
        size += 4.0 * values                                           # the probabilities are part of the result
    return {"flops": flops, "bytes": size}


def _work_train(case):
    cfg = harness.task_config(case["task"], case["B"], native=True, dtype=case["dtype"])
    dim, hid, layers = float(cfg["transformer_dim"]), float(cfg["transformer_hidden_dim"]), cfg["num_layers"]
    tokens = float(case["B"]) * case["L"] * (2 if cfg["dual"] else 1)
    e = 2 if case["dtype"] == "bf16" else 4
    density = {0.8: 0.14, 0.9: 0.10, 0.95: 0.07}.get(case["q"], 0.10)      # typical of discovered masks at this quantile
    flops = layers * (12.0 * density * case["L"] * tokens * dim + 3.0 * tokens * (8.0 * dim * dim + 4.0 * dim * hid))
    # per layer: the attention operands of both directions, the residual stream in and out of both directions, the hidden
    # activation of the feed-forward part written once and read once
    size = layers * tokens * (12.0 * dim * e + 4.0 * dim * 4 + 2.0 * hid * e) + 8.0 * tokens
    return {"flops": flops, "bytes": size}


def tolerance(case):
    kind = case["kind"]
    if kind == "pattern":
        # the masks and block structures are whole numbers; the pooled map is an fp64 sum rounded to fp32 once
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
    if case["dtype"] == "bf16":
        # operands and results rounded to 8 bits, chains of a handful of such roundings
        return {"rel": 1.5e-2} if kind != "train" else {"rel": 2e-2}
    return {"rel": 2e-5} if kind != "train" else {"rel": 1e-4}
