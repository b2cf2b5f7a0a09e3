"""Tangents, conjugate bits and transforms at the entries that pass tensor operations or an autograd function by."""
import pytest
import torch
import torch.autograd.forward_ad as fw

import ash

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("grad_mode", [True, False])
@pytest.mark.parametrize("what", ["beta", "table"])
def test_renderer_refuses_tangents(grad_mode, what):
    """The renderer has no forward-mode derivative: it says so instead of dropping the tangent."""
    from ash.render import render_rays

    grid = ash.BoundedSparseDenseGrid(3, 27, 4, grid_dim=4, sparse_grid_dim=3, device=DEV)
    grid.dense_init_()
    grid.embeddings.requires_grad_(False)
    beta = torch.tensor([0.1], device=DEV)
    o, d = torch.zeros(5, 3, device=DEV), torch.nn.functional.normalize(torch.ones(5, 3, device=DEV), dim=-1)
    with fw.dual_level(), torch.set_grad_enabled(grad_mode):
        render_rays(grid, o, d, 0.0, 1.0, 8, beta)          # nothing carries a tangent
        if what == "beta":
            beta = fw.make_dual(beta, torch.ones_like(beta))
        else:
            dual = fw.make_dual(grid.embeddings.detach(), torch.ones_like(grid.embeddings))
            del grid.embeddings
            grid.embeddings = dual
        with pytest.raises(RuntimeError, match="jvp"):
            render_rays(grid, o, d, 0.0, 1.0, 8, beta)
