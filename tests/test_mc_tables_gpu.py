"""The triangle passes at block edges of every kind of tile (several blocks a tile, byte-wise requests, one
block a tile, beyond the staged edge), on lists that end inside a tile, on blocks without their upper
neighbours, and with cell tables in another order of the cells: against the CPU oracle, exactly."""
import pytest
import torch

from test_mc_gpu import _compare_with_oracle

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _noisy_grid(G, side, spare):
    import ash

    n = side**3
    grid = ash.UnBoundedSparseDenseGrid(3, n + spare, 1, G, cell_size=0.1, device=DEV)
    r = torch.arange(-(side // 2), side - side // 2, device=DEV, dtype=torch.int32)
    coords = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).view(-1, 3)
    grid.engine.insert_keys(coords[torch.arange(n, device=DEV) % 7 != 3].contiguous())   # holes in the lattice
    grid.construct_grid_neighbor_lut_(1, False)
    gen = torch.Generator(device=DEV).manual_seed(G)
    shape = (n + spare, G**3)
    return grid, torch.randn(shape, generator=gen, device=DEV), torch.rand(shape, generator=gen, device=DEV) + 0.97


@pytest.mark.parametrize("G,side,spare", [(1, 5, 0), (2, 5, 3), (3, 4, 1), (4, 4, 0), (5, 3, 2), (6, 3, 0), (7, 3, 0),
                                          (8, 3, 5), (16, 2, 0), (17, 2, 1)])
def test_block_edges(G, side, spare):
    grid, sdf, w = _noisy_grid(G, side, spare)
    sdf.view(-1)[::97] = 0.1   # on the surface
    w.view(-1)[::501] = float("inf")
    _compare_with_oracle(grid, sdf, w, 0.1, 1.0)


@pytest.mark.parametrize("G", [3, 4, 8])
def test_cells_in_another_order(G):
    grid, sdf, w = _noisy_grid(G, 3, 0)
    order = torch.randperm(G**3, generator=torch.Generator().manual_seed(1)).to(DEV)   # new cell i is old cell order[i]
    name = torch.empty_like(order)
    name[order] = torch.arange(G**3, device=DEV)
    grid.cell_coords = grid.cell_coords[order].contiguous()
    grid.lut_cell_nb2cell_idx = name[grid.lut_cell_nb2cell_idx[order]].contiguous()
    grid.lut_cell_nb2grid_nb = grid.lut_cell_nb2grid_nb[order].contiguous()
    _compare_with_oracle(grid, sdf, w, 0.0, 1.0)


def test_a_list_of_some_blocks():
    import __ash
    import numpy as np
    import oracle

    grid, sdf, w = _noisy_grid(8, 3, 0)
    _, idx = grid.engine.items()
    tables = (idx[:11].contiguous(), grid.grid_coords, grid.lut_grid_nb2grid_idx, grid.cell_coords,
              grid.lut_cell_nb2cell_idx, grid.lut_cell_nb2grid_nb)
    mesh = __ash.marching_cubes(sdf, w, *tables, 8, 0.0, 1.0)
    ref = oracle.marching_cubes(sdf.cpu().numpy(), w.cpu().numpy(), *[t.cpu().numpy() for t in tables], 8, 0.0, 1.0)
    assert mesh[0].shape[0] == ref[0].shape[0]
    # vertices owned by a block outside the list are not placed: their id is -1 on both sides
    np.testing.assert_array_equal(np.sort((mesh[0] < 0).sum(1).cpu().numpy()), np.sort((ref[0] < 0).sum(1)))


@pytest.mark.parametrize("G", [3, 8])
def test_a_block_listed_twice(G):
    """Its triangles come twice, its vertices once: every id points at a vertex that was placed."""
    import __ash
    import mesh_checks
    import numpy as np

    grid, sdf, w = _noisy_grid(G, 3, 0)
    _, idx = grid.engine.items()
    rest = (grid.grid_coords, grid.lut_grid_nb2grid_idx, grid.cell_coords, grid.lut_cell_nb2cell_idx,
            grid.lut_cell_nb2grid_nb, G, 0.0, 1.0)
    tris, verts = [t.cpu().numpy() for t in __ash.marching_cubes(sdf, w, idx, *rest)]
    tris2, verts2 = [t.cpu().numpy() for t in __ash.marching_cubes(sdf, w, torch.cat([idx, idx]), *rest)]
    assert verts2.shape == verts.shape and tris2.shape[0] == 2 * tris.shape[0]
    assert tris2.min() >= 0 and tris2.max() < verts.shape[0]
    np.testing.assert_array_equal(verts2[np.lexsort(verts2.T[::-1])], verts[np.lexsort(verts.T[::-1])])
    np.testing.assert_array_equal(mesh_checks.canonical_triangle_rows(verts2, tris2),
                                  np.repeat(mesh_checks.canonical_triangle_rows(verts, tris), 2, axis=0))


@pytest.mark.parametrize("G,side", [(4, 26), (6, 17), (8, 14), (16, 11), (17, 4)])
def test_more_tiles_than_ctas(G, side):
    """Six CTAs per SM share out the tiles (beyond the staged edge: 256 cells at a time), so each takes more than one."""
    grid, sdf, w = _noisy_grid(G, side, 1)
    _compare_with_oracle(grid, sdf + 2.5, w, 0.0, 1.0)


@pytest.mark.parametrize("G", [4, 8, 16])
def test_values_off_their_alignment(G):
    """Rows of cells that start where wide loads may not."""
    grid, sdf, w = _noisy_grid(G, 3, 1)
    shift = lambda t: torch.cat([t.new_zeros(1), t.view(-1)])[1:].view(t.shape)
    _compare_with_oracle(grid, shift(sdf), shift(w), 0.1, 1.0)
