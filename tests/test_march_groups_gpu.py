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


@pytest.mark.parametrize("cell_size", [0.02, 1.0 / 3.0, 7e-4])
@pytest.mark.parametrize("n", [0, 1, 85, 1000])
def test_rays_to_cells_rounds_as_the_tensor_expressions(cell_size, n):
    import __ash

    g = torch.Generator(device=DEV).manual_seed(n)
    o = torch.randn(n, 3, device=DEV, generator=g)
    lo, hi = torch.randn(2, 3, device=DEV, generator=g)
    origin = [float(v) for v in torch.randn(3, generator=g, device=DEV)]
    shift = torch.tensor(origin, device=DEV)
    for got, x in zip(__ash.rays_to_cells(o, lo, hi, origin, cell_size), (o, lo, hi)):
        assert torch.equal(got, (x - shift) / cell_size)


@pytest.mark.parametrize("parallel", [False, True])
def test_outputs_take_gradients_of_any_layout_and_may_be_changed_in_place(parallel):
    from ash.render import render_rays
    from test_raymarch_gpu import make_grid

    grid = make_grid("bounded", 4, seed=5)
    o, d = make_rays(grid, 300, 3, torch.zeros(3, device=DEV))
    coef = torch.randn(3, 300, device=DEV).t()
    grads = []
    for dense in (False, True):
        grid.embeddings.grad = None
        beta = torch.tensor([0.03], device=DEV, requires_grad=True)
        out = render_rays(grid, o, d, 0.05, 2.0, 48, beta, parallel_samples=parallel)
        assert not any(out[k].requires_grad for k in ("n_samples", "near", "far"))
        if dense:
            (out["rgb"] * coef.contiguous() + out["weights"] * torch.ones_like(out["weights"])).sum().backward()
        else:
            out["rgb"].mul_(coef).add_(out["weights"])
            out["rgb"].sum().backward()
        grads.append((grid.embeddings.grad.clone(), beta.grad.clone()))
    scale = float(grads[1][0].abs().max())
    torch.testing.assert_close(grads[0][0], grads[1][0], rtol=1e-4, atol=1e-5 * scale)
    torch.testing.assert_close(grads[0][1], grads[1][1], rtol=1e-4, atol=1e-6)
