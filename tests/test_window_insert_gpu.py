"""Batches that are sorted by table window before they are inserted: the same keys end up in the map, each once
and with an index of its own, as after the insertion in the batch's order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _unique(keys):
    return torch.unique(keys, dim=0)


@pytest.mark.parametrize("dim,n,spread", [(3, 2_100_001, 2**18), (2, 2_097_152, 2**12), (1, 3_000_001, 2**30), (3, 4_000_000, 40)])
def test_sorted_insert(dim, n, spread):
    import __ash
    import ash

    m = ash.HashSet(dim, 5_000_000, DEV)      # 2^24 slots: the smallest table that is sorted for
    ws = __ash._lib.ashb_map_insert_workspace
    h = m.engine.backend._h
    assert ws(h, n) > 0 and ws(h, 2_097_151) == 0
    g = torch.Generator(device=DEV).manual_seed(n)
    keys = torch.randint(-spread, spread, (n, dim), generator=g, device=DEV, dtype=torch.int32)
    keys[n // 2:n // 2 + 1000] = keys[:1000]                   # some twice, and (spread 40) all many times over
    present = keys[: n // 10].contiguous()
    m.insert(present)                                         # a small batch: in its own order
    first = dict(zip(("masks", "rows"), m.engine.find(present)[::-1]))
    m.insert(keys)
    want = _unique(keys)
    got, rows = m.engine.items()
    assert torch.equal(_unique(got), want) and got.shape == want.shape
    assert torch.equal(torch.sort(rows).values, torch.arange(want.shape[0], device=DEV))
    rows_now, masks = m.engine.find(present)
    assert bool(masks.all()) and bool(first["masks"].all()) and torch.equal(rows_now, first["rows"])   # kept their rows
    assert bool(m.find(keys).all())
    absent = keys.clone()
    absent[:, 0] += 2 * spread if spread < 2**20 else 0
    if spread < 2**20:
        assert not bool(m.find(absent).any())
    m.erase(want[::2].contiguous())
    mask = m.find(want)
    assert not bool(mask[::2].any()) and bool(mask[1::2].all())
    m.insert(keys)                                            # over tombstones
    got, rows = m.engine.items()
    assert got.shape == want.shape and torch.unique(rows).numel() == want.shape[0]


def test_sorted_insert_beyond_capacity_reports_and_keeps_what_fits():
    import ash

    m = ash.HashSet(3, 4_300_000, DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    keys = torch.randint(-2**18, 2**18, (5_000_000, 3), generator=g, device=DEV, dtype=torch.int32)
    with pytest.warns(UserWarning):
        m.insert(keys)
    assert m.size() == 4_300_000 and int(m.find(keys).sum()) >= 4_300_000


@pytest.mark.parametrize("capacity", [1000, 5_000_000])
@pytest.mark.parametrize("dim", [1, 2, 3, 4])
def test_contains_is_the_masks_of_find(capacity, dim):
    import __ash
    import ash

    m = ash.HashSet(dim, capacity, DEV)
    g = torch.Generator(device=DEV).manual_seed(dim)
    keys = torch.randint(-300, 300, (999, dim), generator=g, device=DEV, dtype=torch.int32)
    m.insert(keys[:500].contiguous())
    for coop in (False, True):
        __ash.set_find_cooperative(coop)
        try:
            assert torch.equal(m.find(keys), m.engine.find(keys)[1])
        finally:
            __ash.set_find_cooperative(False)
