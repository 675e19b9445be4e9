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
