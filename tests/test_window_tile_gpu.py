"""Sorted insertion of batches whose keys start where wide loads may not, and that end inside a tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dim,skip,tail", [(1, 0, 0), (1, 1, 1), (1, 3, 2047), (2, 1, 5), (2, 2, 0), (3, 0, 1), (3, 1, 0), (3, 2, 100),
                                           (3, 3, 2047)])
def test_offset_and_ragged_batches(dim, skip, tail):
    import ash

    capacity = 33_554_432                                   # 2^26 slots: a table of 1 GB
    n = capacity // 4 + tail                                # a key per 128-byte line, tiles of 2048 and a rest
    i = torch.randperm(n + skip, device=DEV)
    keys = torch.stack([i % 65_536, i // 65_536, -i], 1)[:, :dim] if dim > 1 else i.view(-1, 1)
    keys = keys.to(torch.int32).contiguous()[skip:]
    assert keys.is_contiguous() and keys.shape == (n, dim)
    s = ash.HashSet(dim, capacity, DEV)
    s.insert(keys)
    assert s.size() == n and s.find(keys).all()
    assert not s.find(keys + 100_000_000).any()
    rows = s.engine.find(keys)[0]
    assert torch.unique(rows).numel() == n and int(rows.max()) == n - 1     # a row each, the first n of the stack
    assert s.engine.backend.status() == 0
