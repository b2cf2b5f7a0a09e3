"""What ``gaussian_filter_`` owes its caller besides the values."""
import pytest
import torch

import ash

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _grid(G=4, D=2, n=20, spare=5, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    cells = torch.randperm(27, generator=g, device=DEV)[:n]
    grid = ash.SparseDenseGrid(3, n + spare, D, G, DEV)
    grid.engine.insert_keys(torch.stack([cells % 3, cells // 3 % 3, cells // 9], 1).int())
    grid.embeddings.data.normal_(generator=g)
    grid.construct_grid_neighbor_lut_(1, False)
    return grid


@pytest.mark.parametrize("separable", [True, False])
def test_backward_after_the_filter_is_refused(separable):
    """A forward pass has saved the table for its backward; filtered in between it is another table."""
    grid = _grid()
    grid.separable_gaussian = separable
    x = (torch.rand(50, 3, device=DEV) * 8).requires_grad_(True)
    y, _ = grid(x)
    grid.gaussian_filter_(3, 1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


def test_render_backward_after_the_filter_is_refused():
    from ash.render import render_rays

    grid = _grid(D=4)
    grid.bbox_min, grid.bbox_max = torch.zeros(3, device=DEV), torch.full((3,), 12.0, device=DEV)
    grid.cell_size = 1.0
    o = torch.rand(20, 3, device=DEV) * 10
    d = torch.nn.functional.normalize(torch.randn(20, 3, device=DEV), dim=-1)
    out = render_rays(grid, o, d, 0.0, 20.0, 16, torch.tensor([0.5], device=DEV))
    grid.gaussian_filter_(3, 1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out["rgb"].sum().backward()


@pytest.mark.parametrize("rows", [12, 40])
def test_table_of_another_row_count_is_refused(rows):
    """Rows of a shard are not the map's indices."""
    grid = _grid(n=20, spare=5)
    grid.embeddings = torch.nn.Parameter(torch.randn(rows, 64, 2, device=DEV))
    before = grid.embeddings.detach().clone()
    with pytest.raises(RuntimeError):
        grid.gaussian_filter_(3, 1.0)
    assert torch.equal(grid.embeddings.detach(), before)


def test_other_strides_are_filtered_too():
    grid = _grid()
    start = grid.embeddings.detach().clone()
    grid.gaussian_filter_(5, 1.5)
    want = grid.embeddings.detach().clone()
    grid.embeddings = torch.nn.Parameter(start.permute(2, 0, 1).contiguous().permute(1, 2, 0))
    assert not grid.embeddings.is_contiguous()
    grid.gaussian_filter_(5, 1.5)
    assert torch.equal(grid.embeddings.detach(), want)


@pytest.mark.parametrize("call", [lambda g: g.gaussian_filter_(3, 1.0)])
def test_capture_is_refused(call):
    """A graph would hold the address of factors that a later call replaces."""
    grid = _grid()
    call(grid)
    before = grid.embeddings.detach().clone()
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError, match="captur"):
        with torch.cuda.graph(graph):
            call(grid)
    del graph
    torch.cuda.synchronize()
    assert torch.equal(grid.embeddings.detach(), before)
    call(grid)
