"""The renderer's kernels are compiled for tables within and beyond the reach of 32-bit byte offsets: both give the same
rays and gradients.  And the march's shortcut inside the box keeps every step, wherever a ray enters and leaves."""
import numpy as np
import pytest
import torch

from test_raymarch_gpu import make_grid, make_rays

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _spread_over(grid, capacity, D):
    """The same blocks and rows in a table of `capacity` rows, the rows spread over all of it."""
    import ash

    keys, rows = grid.engine.items()
    n = len(keys)
    at = torch.arange(n, device=DEV) * (capacity // n) + capacity % n
    big = ash.UnBoundedSparseDenseGrid(3, capacity, D, 8, cell_size=grid.cell_size, device=DEV)
    heap = torch.arange(capacity, dtype=torch.int32, device=DEV)
    used = torch.zeros(capacity, dtype=torch.bool, device=DEV)
    used[at] = True
    all_keys = torch.zeros((capacity, 3), dtype=torch.int32, device=DEV)
    indices = torch.zeros(capacity, dtype=torch.long, device=DEV)
    all_keys[:n], indices[:n] = keys, at
    big.engine.load_state_dict({"_heap": torch.cat([heap[used], heap[~used]]), "_keys": all_keys, "_indices": indices,
                                "_size": torch.tensor([n], dtype=torch.int32, device=DEV)})
    with torch.no_grad():
        big.embeddings.zero_()
        big.embeddings[at] = grid.embeddings[rows]
    big.construct_grid_neighbor_lut_(radius=1, bidirectional=False)
    return big, rows, at


@pytest.mark.parametrize("interpolation", ["linear", "smooth_step"])
@pytest.mark.parametrize("parallel", [False, True])
def test_offsets_of_both_widths(interpolation, parallel):
    from ash.render import render_rays

    small = make_grid("unbounded", 4, 9)
    big, rows, at = _spread_over(small, 540_000, 4)     # 4.4 GB: the last rows lie beyond 2^32 bytes
    assert big.embeddings.numel() * 4 > 2**32
    o, d = make_rays(small, 1000, 2, torch.tensor([0.3, -0.2, 0.1], device=DEV))
    outs, grads = [], []
    for grid in (small, big):
        beta = torch.tensor([0.04], device=DEV, requires_grad=True)
        # one box for both: the marches go through the same sums
        grid.bbox_min, grid.bbox_max = small.bbox_min, small.bbox_max
        out = render_rays(grid, o, d, 0.1, 2.5, 48, beta, interpolation, parallel_samples=parallel)
        (out["rgb"].sum() + out["depth"].sum() + out["normal"][:, 0].sum()).backward()
        outs.append(out)
        grads.append((grid.embeddings.grad, beta.grad))
    assert outs[0]["n_samples"].sum() > 5000
    for name in ("near", "far", "n_samples"):
        assert torch.equal(outs[0][name], outs[1][name]), name
    for name in ("rgb", "depth", "normal", "weights", "eikonal_l2"):
        # the same products; a sum may be contracted differently: 48 samples of 8 terms
        scale = outs[0][name].abs().max()
        assert (outs[0][name] - outs[1][name]).abs().max() <= 48 * 8 * 2**-24 * scale, name
    ga, gb = grads[0][0][rows], grads[1][0][at]
    assert (ga - gb).abs().max() <= 1e-4 * ga.abs().max()      # atomic sums in any order, cancelling
    rest = torch.ones(len(big.embeddings), dtype=torch.bool, device=DEV)
    rest[at] = False
    assert not big.embeddings.grad[rest].any()


def test_box_of_any_place():
    """Rays that start outside the box, inside it near a face, run along a face, or never move along an axis."""
    import oracle

    grid = make_grid("unbounded", 4, 4)
    cs = grid.cell_size
    om = oracle.OracleHashMap(3, 6000)
    om.insert_keys(grid.engine.items()[0].cpu().numpy())
    g = torch.Generator(device=DEV).manual_seed(1)
    n = 4000
    grid.compute_bbox_()
    lo, hi = grid.bbox_min, grid.bbox_max
    lo, hi = lo + 0.3 * (hi - lo), hi - 0.2 * (hi - lo)          # a box that cuts through the blocks
    o = lo + (hi - lo) * (torch.rand(n, 3, generator=g, device=DEV) * 1.6 - 0.3)
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV), dim=-1)
    d[::7, 1] = 0.0
    d[::11, :2] = 0.0
    o[::5, 0] = hi[0]
    o[1::5, 2] = lo[2]
    import __ash

    args = (o / cs, d, lo / cs, hi / cs)
    nears, fars = __ash.ray_find_near_far(grid.engine.backend, *args, 0.0, 2.5 / cs, 0.01 / cs, 8.0)
    n_ref, f_ref = oracle.ray_find_near_far(om, *[a.cpu().numpy() for a in args], 0.0, 2.5 / cs, 0.01 / cs, 8.0)
    assert (n_ref >= 0).sum() > 500 and (n_ref < 0).sum() > 500
    np.testing.assert_array_equal(nears.cpu().numpy().reshape(-1), n_ref.reshape(-1))
    np.testing.assert_array_equal(fars.cpu().numpy().reshape(-1), f_ref.reshape(-1))
