"""Batches that are sorted by table window before they are inserted: the same keys end up in the map, each once
and with an index of its own, as after the insertion in the batch's order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _packed(keys):
    p = torch.zeros(keys.shape[0], dtype=torch.int64, device=DEV)
    for d in range(keys.shape[1]):
        p = p * 2**20 + keys[:, d].long() + 2**19 if keys.shape[1] > 1 else keys[:, 0].long()
    return p


CAPACITY = 16_777_217     # 2^26 slots: the smallest table that is sorted for, from a key per line on


@pytest.mark.parametrize("dim,n,spread", [(3, 8_388_609, 2**18), (2, 8_388_608, 2**12), (1, 12_000_001, 2**30), (3, 9_000_000, 40)])
def test_sorted_insert(dim, n, spread):
    import __ash
    import ash

    m = ash.HashSet(dim, CAPACITY, DEV)
    ws = __ash._lib.ashb_map_insert_workspace
    h = m.engine.backend._h
    assert ws(h, n) > 0 and ws(h, 8_388_607) == 0
    g = torch.Generator(device=DEV).manual_seed(n)
    keys = torch.randint(-spread, spread, (n, dim), generator=g, device=DEV, dtype=torch.int32)
    keys[n // 2:n // 2 + 1000] = keys[:1000]                   # some twice, and (spread 40) all many times over
    present = keys[: n // 10].contiguous()
    m.insert(present)                                         # a small batch: in its own order
    rows_before, masks_before = m.engine.find(present)
    m.insert(keys)
    order = torch.sort(_packed(keys), stable=True)
    firsts = torch.ones(n, dtype=torch.bool, device=DEV)
    firsts[1:] = order.values[1:] != order.values[:-1]
    want = keys[order.indices[firsts]].contiguous()           # each distinct key once
    got, rows = m.engine.items()
    assert torch.equal(torch.sort(_packed(got)).values, _packed(want))
    assert torch.equal(torch.sort(rows).values, torch.arange(want.shape[0], device=DEV))
    rows_now, masks = m.engine.find(present)
    assert bool(masks.all()) and bool(masks_before.all()) and torch.equal(rows_now, rows_before)   # kept their rows
    assert bool(m.find(keys).all())
    if spread < 2**20:
        absent = keys.clone()
        absent[:, 0] += 2 * spread
        assert not bool(m.find(absent).any())
    m.erase(want[::2].contiguous())
    mask = m.find(want)
    assert not bool(mask[::2].any()) and bool(mask[1::2].all())
    m.insert(keys)                                            # over tombstones
    got, rows = m.engine.items()
    assert torch.equal(torch.sort(_packed(got)).values, _packed(want)) and torch.unique(rows).numel() == want.shape[0]


def test_sorted_insert_beyond_capacity_reports_and_keeps_what_fits():
    import ash

    m = ash.HashSet(3, CAPACITY, DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    keys = torch.randint(-2**18, 2**18, (18_000_000, 3), generator=g, device=DEV, dtype=torch.int32)
    with pytest.warns(UserWarning):
        m.insert(keys)
    assert m.size() == CAPACITY and int(m.find(keys).sum()) >= CAPACITY


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


@pytest.mark.parametrize("capacity", [700, 3_000_000])      # without and with the occupancy bits asked first
@pytest.mark.parametrize("dim", [1, 3, 4])
def test_find_with_values_is_find_and_indexing(capacity, dim):
    import ash

    m = ash.HashMap(dim, {"a": 1, "b": 3, "c": 16, "wide": 40}, capacity, DEV)
    g = torch.Generator(device=DEV).manual_seed(dim)
    keys = torch.randint(-9, 9, (701, dim), generator=g, device=DEV, dtype=torch.int32)
    values = {k: torch.randn(701, w, generator=g, device=DEV) for k, w in m.value_dims.items()}
    m.insert(keys[:600].contiguous(), {k: v[:600].contiguous() for k, v in values.items()})
    for n in (701, 1, 0):
        if n == 0:
            with pytest.warns(UserWarning):
                masks, idx, got = m.find(keys[:0], return_values=True)
        else:
            masks, idx, got = m.find(keys[:n], return_values=True)
        assert got.keys() == values.keys() and got["b"].shape == (n, 3)
        ref_idx, ref_masks = (idx, masks) if n == 0 else m.engine.find(keys[:n])
        assert torch.equal(idx, ref_idx) and torch.equal(masks, ref_masks)
        for k, v in m.values.items():
            assert torch.equal(got[k], v[ref_idx]), k
    backend = m.engine.backend
    odd = {"bytes": torch.randint(0, 255, (capacity, 3), device=DEV, dtype=torch.uint8), "d": torch.randn(capacity, 2, device=DEV).double(),
           "flat": torch.arange(capacity, device=DEV, dtype=torch.int16)}
    idx, masks, got = backend.find_values(keys, odd)
    for k, v in odd.items():
        assert got[k].dtype == v.dtype and torch.equal(got[k], v[idx]), k
    assert backend.find_values(keys, {"wide": m.values["wide"]}) is None
    assert backend.find_values(keys, {"p": torch.zeros(capacity, 1, device=DEV, requires_grad=True)}) is None


@pytest.mark.parametrize("capacity", [1, 5, 1000, 1_000_000, 3_000_000])
@pytest.mark.parametrize("dim", [2, 4])
def test_clear_leaves_an_empty_map(capacity, dim):
    import ash

    m = ash.HashSet(dim, capacity, DEV)
    n = min(capacity, 2000)
    keys = torch.arange(n * dim, device=DEV, dtype=torch.int32).view(n, dim)
    for _ in range(2):
        m.insert(keys)
        assert m.size() == n and bool(m.find(keys).all())
        m.clear()
        assert m.size() == 0 and not bool(m.find(keys).any()) and m.keys().shape[0] == 0
        assert torch.equal(m.engine._heap, torch.arange(capacity, device=DEV, dtype=torch.int32))


@pytest.mark.parametrize("batch,sorts", [("distinct", True), ("half of them twice", True), ("one key", False), ("runs of twelve", False),
                                         ("few in any order", False)])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_batches_of_repeats_go_in_their_own_order(batch, sorts, dim):
    """The window counts at the workspace's head stay zero where the sample finds too few distinct keys."""
    import __ash
    import ash

    n = 9_000_001
    m = ash.HashSet(dim, CAPACITY, DEV)
    g = torch.Generator(device=DEV).manual_seed(dim)
    span = {1: 2**30, 2: 2**19, 3: 2**18}[dim]
    keys = torch.randint(-span, span, (n, dim), generator=g, device=DEV, dtype=torch.int32)
    if batch == "half of them twice":
        keys[n // 2:] = keys[torch.randint(n // 2, (n - n // 2,), generator=g, device=DEV)]
        keys = keys[torch.randperm(n, generator=g, device=DEV)]
    elif batch == "one key":
        keys[:] = keys[0]
    elif batch == "runs of twelve":
        keys = keys[torch.arange(n, device=DEV) // 12]
    elif batch == "few in any order":
        keys = keys[torch.randint(100_000, (n,), generator=g, device=DEV)]
    keys = keys.contiguous()
    h, stream = m.engine.backend._h, torch.cuda.current_stream().cuda_stream
    workspace = torch.empty(__ash._lib.ashb_map_insert_workspace(h, n) // 4, dtype=torch.int32, device=DEV)
    assert __ash._lib.ashb_map_insert_keys_sorted(h, keys.data_ptr(), n, workspace.data_ptr(), workspace.numel() * 4, stream) == 0
    assert int(workspace[:256].sum()) == (n if sorts else 0)
    got, rows = m.engine.items()
    want = torch.unique(_packed(keys))
    assert torch.equal(torch.sort(_packed(got)).values, want)
    assert torch.equal(torch.sort(rows).values, torch.arange(want.shape[0], device=DEV))


def test_rows_of_many_small_words_are_left_to_indexing():
    import ash

    m = ash.HashMap(3, 1, 500, DEV)
    keys = torch.randint(-9, 9, (300, 3), device=DEV, dtype=torch.int32)
    m.engine.insert_keys(keys)
    find, bytes_of = m.engine.backend.find_values, lambda w: torch.randint(0, 255, (500, w), device=DEV, dtype=torch.uint8)
    unaligned = bytes_of(32).view(-1).new_zeros(500 * 32 + 1)[1:].view(500, 32)
    for table, gathers in ((bytes_of(15), True), (bytes_of(17), False), (bytes_of(32), True), (bytes_of(30), True), (bytes_of(34), False),
                           (bytes_of(60), True), (bytes_of(64), True), (bytes_of(68), False), (unaligned, False)):
        found = find(keys, {"t": table})
        assert (found is not None) == gathers, table.shape
        m.values["default"] = table
        _, rows, got = m.find(keys, return_values=True)
        assert torch.equal(got, table[rows])


@pytest.mark.parametrize("route", ["no memory", "side stream"])
def test_sorted_insert_without_its_workspace_and_on_a_side_stream(route, monkeypatch):
    import ash

    m = ash.HashSet(3, CAPACITY, DEV)
    g = torch.Generator(device=DEV).manual_seed(11)
    keys = torch.randint(-2**18, 2**18, (8_500_000, 3), generator=g, device=DEV, dtype=torch.int32)
    want = torch.unique(_packed(keys))
    empty, refused = torch.empty, []

    def no_workspace(*args, **kwargs):
        if route == "no memory" and kwargs.get("dtype") is torch.uint8:
            refused.append(args)
            raise torch.cuda.OutOfMemoryError("no room for the workspace")
        return empty(*args, **kwargs)

    side = torch.cuda.Stream() if route == "side stream" else torch.cuda.current_stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), monkeypatch.context() as patch:
        patch.setattr(torch, "empty", no_workspace)
        m.insert(keys)
        # the workspace's memory goes to whoever asks next on this stream, after the insertion
        empty(sum(keys.shape) * 12, dtype=torch.uint8, device=DEV).fill_(255)
    side.synchronize()
    assert len(refused) == (route == "no memory")
    got, rows = m.engine.items()
    assert torch.equal(torch.sort(_packed(got)).values, want)
    assert torch.equal(torch.sort(rows).values, torch.arange(want.shape[0], device=DEV))
