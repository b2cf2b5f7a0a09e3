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
