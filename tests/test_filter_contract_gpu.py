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


def _overflow(grid):
    keys = torch.arange(30, dtype=torch.int32, device=DEV).view(-1, 1).repeat(1, 3)
    grid.engine.backend.insert_keys(keys)        # as native insertions do: past the host's own bound


@pytest.mark.parametrize("call", [lambda g: g.gaussian_filter_(3, 1.0), lambda g: g.construct_grid_neighbor_lut(1, True)])
def test_dropped_keys_are_reported(call):
    grid = _grid()
    _overflow(grid)
    with pytest.warns(UserWarning, match="capacity"):
        call(grid)


def test_a_table_in_error_is_left_unfiltered():
    grid = _grid()
    keys, index = grid.engine.items()
    keys[1] = keys[0]
    import __ash

    h = grid.engine.backend
    rc = __ash._lib.ashb_map_load_states(h._h, keys.data_ptr(), index.data_ptr(), keys.shape[0], h._heap.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    before = grid.embeddings.detach().clone()
    with pytest.raises(RuntimeError, match="status"):
        grid.gaussian_filter_(3, 1.0)
    assert torch.equal(grid.embeddings.detach(), before)


@pytest.mark.parametrize("call", [lambda g: g.gaussian_filter_(3, 1.0), lambda g: g.construct_grid_neighbor_lut(1, True)])
def test_capture_is_refused(call):
    """The call reads the map's status, and a graph would hold the address of factors that a later call replaces."""
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


def test_window_kept_by_another_thread_is_not_used():
    """Another thread's window may take the place of this call's at any time."""
    grid, alone = _grid(seed=4), _grid(seed=4)
    alone.gaussian_filter_(3, 1.0)
    ours = alone._gaussian_window
    other = _grid(seed=4)
    other.gaussian_filter_(3, 2.0)
    theirs, start = other._gaussian_window, grid.embeddings.detach().clone()
    for looks in range(4):
        class Raced(ash.SparseDenseGrid):
            seen = 0

            @property
            def _gaussian_window(self):
                Raced.seen += 1
                return ours if Raced.seen <= looks else theirs

            @_gaussian_window.setter
            def _gaussian_window(self, value):
                pass

        grid.embeddings.data.copy_(start)
        grid.__class__ = Raced
        grid.gaussian_filter_(3, 1.0)
        grid.__class__ = ash.SparseDenseGrid
        want = grid.embeddings.detach().clone()
        grid.embeddings.data.copy_(start)
        grid.gaussian_filter_(3, 1.0)
        assert torch.equal(want, grid.embeddings.detach()), looks


@pytest.mark.parametrize("G,size,D,side,spare", [(4, 3, 1, 28, 100), (8, 7, 4, 17, 3000), (16, 7, 4, 11, 1), (5, 5, 13, 11, 200),
                                                 (3, 3, 1, 20, 0)])
def test_more_blocks_than_ctas(G, size, D, side, spare):
    """Beyond eight waves of CTAs each takes a second block (and a second row to copy back): the same bits as with a CTA per
    block, and zeros in the spare rows."""
    import __ash as native

    n = side**3
    cells = torch.arange(n, device=DEV)
    cells = cells[cells % 7 != 3]                                   # holes in the lattice
    grid = ash.SparseDenseGrid(3, len(cells) + spare, D, G, DEV)
    grid.engine.insert_keys(torch.stack([cells % side, cells // side % side, cells // side**2], 1).int())
    grid.embeddings.data.normal_(generator=torch.Generator(device=DEV).manual_seed(G))
    _, lut = grid.construct_grid_neighbor_lut(1, bidirectional=True)
    _, index = grid.engine.items()
    start = grid.embeddings.detach().clone()
    grid.gaussian_filter_(size, 1.5)
    want = native.convolution_forward_separable(start, grid._gaussian_window[1], index.view(-1, 1), lut, G, size // 2)
    assert torch.equal(grid.embeddings.detach(), want)
    rest = torch.ones(len(cells) + spare, dtype=torch.bool, device=DEV)
    rest[index] = False
    assert int(rest.sum()) == spare and not bool(want[rest].any())


def test_windows_replaced_on_another_stream():
    grid = _grid(D=16, seed=5)
    start = grid.embeddings.detach().clone()
    for _ in range(20):
        grid.gaussian_filter_(3, 1.0)
        grid.gaussian_filter_(5, 2.0)
    want = grid.embeddings.detach().clone()
    grid.embeddings.data.copy_(start)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(20):
            grid.gaussian_filter_(3, 1.0)
            grid.gaussian_filter_(5, 2.0)
            torch.full((3, 3, 16), 7.0, device=DEV), torch.full((3, 5, 16), 7.0, device=DEV)   # into what was given back
    side.synchronize()
    assert torch.equal(grid.embeddings.detach(), want)
