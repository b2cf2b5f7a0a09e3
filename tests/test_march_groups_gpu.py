"""The march by a group of lanes per ray against the march by one thread per ray: near, far and the number of
intervals must be the same numbers, for batches that end inside a warp, ranges that start behind the origin,
ranges of less than a step, rays with many intervals, and tables beyond the size whose occupancy bits are
asked first."""
import pytest
import torch

from test_raymarch_gpu import DEV, make_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [6000, 300_000])
@pytest.mark.parametrize("n,t_min,t_max,samples", [(1, 0.05, 2.0, 48), (33, 0.0, 3.0, 128), (257, -1.0, 2.0, 16), (100, 0.3, 0.301, 48),
                                                   (500, 0.05, 2.0, 1000), (64, 1.0, 0.5, 48)])
def test_group_march_equals_thread_march(capacity, n, t_min, t_max, samples):
    import ash
    from ash.render import render_rays

    g = torch.Generator(device=DEV).manual_seed(7)
    grid = ash.BoundedSparseDenseGrid(3, capacity, 4, grid_dim=2, sparse_grid_dim=64, device=DEV)
    grid.spatial_init_(torch.nn.functional.normalize(torch.randn(4000, 3, device=DEV, generator=g), dim=-1) * 0.5, dilation=0)
    grid.embeddings.data.normal_(0.0, 0.01, generator=g)
    o, d = make_rays(grid, n, n, torch.zeros(3, device=DEV))
    d[: n // 4, 1] = 0.0                                   # along a face of the lattice
    beta = torch.tensor([0.02], device=DEV)
    with torch.no_grad():
        thread = render_rays(grid, o, d, t_min, t_max, samples, beta, parallel_samples=False)
        group = render_rays(grid, o, d, t_min, t_max, samples, beta, parallel_samples=True)
    for k in ("near", "far", "n_samples"):
        assert torch.equal(thread[k], group[k]), k
    for k in ("depth", "weights"):
        torch.testing.assert_close(group[k], thread[k], rtol=2e-4, atol=2e-5)
