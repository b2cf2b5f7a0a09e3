"""Queries without a gradient (a miss, an absent neighbour) in the row list: zero rows that point at valid cells."""
import pytest
import torch

import ash

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n_blocks", [1, 37])
@pytest.mark.parametrize("G,D,positions", [(1, 4, False), (2, 16, True), (8, 16, False), (8, 16, True), (8, 5, True), (2, 1, False)])
def test_misses_point_at_valid_cells(G, D, positions, n_blocks):
    g = torch.Generator(device=DEV).manual_seed(G + D)
    grid = ash.SparseDenseGrid(3, n_blocks, D, G, DEV)
    blocks = torch.stack([torch.arange(n_blocks, device=DEV)] * 3, 1).int()
    grid.engine.insert_keys(blocks)
    grid.embeddings.data.normal_(0, 1, generator=g)
    grid.construct_grid_neighbor_lut_(radius=1, bidirectional=False)
    n = 1003
    inside = (blocks[torch.randint(n_blocks, (n,), generator=g, device=DEV)].float() + 0.9 * torch.rand(n, 3, generator=g, device=DEV)) * G
    x = torch.where(torch.rand(n, 1, generator=g, device=DEV) < 0.5, inside, inside + 1000.0 * G)
    z = torch.randn(n, D, generator=g, device=DEV)
    grads = []
    for mode in ("dense", "row_list"):
        grid.grad_mode = mode
        grid.embeddings.grad = None
        xm = x.clone().requires_grad_(positions)
        y, masks = grid(xm, interpolation="linear")
        y.backward(z)
        grads.append((grid.embeddings.grad, xm.grad))
    (dense, gx), (rows, gx_rows) = grads
    idx, values = rows._indices(), rows._values()
    assert rows.is_sparse and idx.shape == (2, 8 * n) and (~masks).any()
    assert (idx >= 0).all() and (idx[0] < n_blocks).all() and (idx[1] < G**3).all()
    assert not values[(~masks).repeat_interleave(8)].any()
    got = torch.zeros_like(dense).index_put_((idx[0], idx[1]), values, accumulate=True)
    # up to 8 n terms of size |z| <= 5 land in a row, in any order
    assert (got - dense).abs().max() <= 8 * n * 2**-24 * values.abs().sum() / max(1, (values != 0).sum()) + 1e-4
    if positions:
        assert torch.equal(gx, gx_rows)
