"""State that the modules keep between calls, as far as it needs no GPU."""
import torch


def test_mask_key_tells_masks_apart():
    """Another view, another type, other contents in the same place, a tensor given other storage: all are other masks."""
    from spion_b200._ops import ops
    key, mat = ops.MaskKey(), torch.eye(4)
    assert not key.matches(mat)
    key.set(mat)
    assert key.matches(mat) and key.matches(mat.view(4, 4))
    assert not key.matches(mat.t()) and not key.matches(mat.view(2, 8)) and not key.matches(mat.view(torch.int32))
    assert not key.matches(mat.clone())
    mat[0, 1] = 1
    assert not key.matches(mat)
    key.set(mat)
    mat.data = torch.ones(4, 4)
    assert not key.matches(mat)
    key.set(mat)
    old = mat.data_ptr()
    mat.data = torch.zeros(4, 4)                        # the key holds on to the storage it names
    others = [torch.empty(4, 4) for _ in range(64)]
    assert all(t.data_ptr() != old for t in others) and not any(key.matches(t) for t in others)


def test_discovery_refuses_maps_of_several_devices():
    """One launch reads all maps of a call."""
    from types import SimpleNamespace

    import pytest

    from spion_b200 import pattern
    maps = [SimpleNamespace(is_cuda=True, device=torch.device("cuda", i)) for i in (0, 1)]
    with pytest.raises(ValueError, match="different devices"):
        pattern._discover(maps, 64, 0.9, "diag", 31, "paths", 0)


def test_a_word_does_not_choose_the_backward_path():
    """recompute is None, False or True; a word ("stored" among them) is refused before anything is created."""
    import pytest

    from spion_b200._lib import SpionError
    from spion_b200.native import BlockSparseAttention
    config = {"head_dim": 32, "num_head": 2, "max_seq_len": 256, "batch_size": 2, "block_size": 64}
    for word in ("stored", "layer", ""):
        with pytest.raises(SpionError, match="recompute must be"):
            BlockSparseAttention(config, dtype=torch.bfloat16, device="cuda:0", recompute=word)


def test_optimizer_state_by_parameter():
    """The state of an optimizer over pieces of the parameters is that of one over the parameters, in both directions."""
    import copy

    from spion_b200.dp import FlatGradBucket

    def model():
        torch.manual_seed(0)
        return torch.nn.Sequential(torch.nn.Embedding(300, 64), torch.nn.Linear(64, 200), torch.nn.Linear(200, 3))

    def steps(m, opt, n, bucket=None):
        g = torch.Generator().manual_seed(n)
        for _ in range(n):
            loss = m(torch.randint(300, (16,), generator=g)).square().mean()
            if bucket is None:
                opt.zero_grad()
                loss.backward()
            else:
                bucket.backward(loss)
            opt.step()

    def pieced(m):
        bucket = FlatGradBucket(m.parameters())
        opt = torch.optim.AdamW(bucket.pieces(), lr=1e-2)
        bucket.state_by_parameter(opt)
        return bucket, opt

    whole, parts = model(), model()
    opt = torch.optim.AdamW(whole.parameters(), lr=1e-2)
    bucket, opt_p = pieced(parts)
    assert len(opt_p.param_groups[0]["params"]) > 5
    assert opt_p.state_dict()["param_groups"][0]["params"] == opt.state_dict()["param_groups"][0]["params"]
    steps(whole, opt, 3)
    steps(parts, opt_p, 3, bucket)
    a, b = copy.deepcopy(opt.state_dict()), copy.deepcopy(opt_p.state_dict())
    assert a["state"].keys() == b["state"].keys()
    for i in a["state"]:
        assert all(torch.equal(a["state"][i][k], b["state"][i][k]) for k in ("step", "exp_avg", "exp_avg_sq"))
    # each goes on from the other's checkpoint
    whole2, parts2 = copy.deepcopy(whole), model()
    parts2.load_state_dict(whole.state_dict())
    opt2 = torch.optim.AdamW(whole2.parameters(), lr=1e-2)
    opt2.load_state_dict(b)
    bucket2, opt_p2 = pieced(parts2)
    opt_p2.load_state_dict(a)
    steps(whole, opt, 2)
    steps(whole2, opt2, 2)
    steps(parts2, opt_p2, 2, bucket2)
    for p, q, r in zip(whole.parameters(), whole2.parameters(), parts2.parameters()):
        assert torch.equal(p, q) and torch.equal(p, r)
