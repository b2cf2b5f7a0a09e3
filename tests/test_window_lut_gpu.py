"""Block-neighbour tables of any radius against a dictionary of the active blocks."""
import itertools

import pytest
import torch

import ash

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,capacity", [(0, 5), (1, 1), (33, 40), (700, 1000)])
@pytest.mark.parametrize("radius,bidirectional", [(0, True), (1, False), (1, True), (2, False), (2, True)])
def test_window_table_equals_dictionary(n, capacity, radius, bidirectional):
    """Exact: coordinates, neighbour rows (x fastest), -1 for absent neighbours and for inactive rows."""
    grid = ash.SparseDenseGrid(3, capacity, 1, 2, DEV)
    g = torch.Generator(device=DEV).manual_seed(n + radius)
    if n:
        cells = torch.randperm(12**3, generator=g, device=DEV)[:n]
        grid.engine.insert_keys((torch.stack([cells % 12, cells // 12 % 12, cells // 144], 1) - 6).int())
    coords, lut = grid.construct_grid_neighbor_lut(radius, bidirectional)
    steps = range(-radius if bidirectional else 0, radius + 1)
    assert coords.dtype == torch.int32 and lut.dtype == torch.int64 and lut.shape == (capacity, len(steps) ** 3)
    keys, index = grid.engine.items()
    rows = {tuple(k): i for k, i in zip(keys.tolist(), index.tolist())}
    want_lut = torch.full(lut.shape, -1, dtype=torch.int64)
    want_coords = torch.full((capacity, 3), -1, dtype=torch.int32)
    for (x, y, z), i in rows.items():
        want_coords[i] = torch.tensor([x, y, z])
        want_lut[i] = torch.tensor([rows.get((x + dx, y + dy, z + dz), -1) for dz, dy, dx in itertools.product(steps, repeat=3)])
    assert torch.equal(coords.cpu(), want_coords) and torch.equal(lut.cpu(), want_lut)


@pytest.mark.parametrize("radius", [64, 65, 70])
def test_wide_one_sided_windows(radius):
    grid = ash.SparseDenseGrid(3, 4, 1, 2, DEV)
    keys = [(0, 0, 0), (radius, 0, 3), (70, 70, 70), (-radius, 1, -2)]
    grid.engine.insert_keys(torch.tensor(keys, dtype=torch.int32, device=DEV))
    coords, lut = grid.construct_grid_neighbor_lut(radius, False)
    keys, index = grid.engine.items()
    S = radius + 1
    want = torch.full((4, S**3), -1, dtype=torch.int64)
    for a, i in zip(keys.tolist(), index.tolist()):
        for b, j in zip(keys.tolist(), index.tolist()):
            dx, dy, dz = (q - p for p, q in zip(a, b))
            if all(0 <= d <= radius for d in (dx, dy, dz)):
                want[i, dx + S * (dy + S * dz)] = j
    assert torch.equal(lut.cpu(), want) and torch.equal(coords[index], keys)
