"""Tangents, conjugate bits and transforms at the entries that pass tensor operations or an autograd function by."""
import pytest
import torch
import torch.autograd.forward_ad as fw

import ash

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _map(dtype=torch.float32):
    m = ash.HashMap(3, 2, 50, DEV)
    keys = torch.randint(-9, 9, (40, 3), dtype=torch.int32, device=DEV)
    m.insert(keys, keys[:, :2].float())
    return m, torch.cat([keys[:20], keys[:5] + 100])


def test_found_values_carry_their_tangent():
    m, q = _map()
    table, tangent = m.values["default"], torch.randn(50, 2, device=DEV)
    with fw.dual_level():
        m.values["default"] = fw.make_dual(table, tangent)
        _, rows, got = m.find(q, return_values=True)
        primal, moved = fw.unpack_dual(got)
        assert torch.equal(primal, table[rows]) and moved is not None and torch.equal(moved, tangent[rows])


def test_found_values_of_conjugated_and_negated_tables():
    m, q = _map()
    for table in (torch.randn(50, 2, dtype=torch.complex64, device=DEV).conj(), torch._neg_view(torch.randn(50, 2, device=DEV))):
        assert table.is_contiguous()
        m.values["default"] = table
        _, rows, got = m.find(q, return_values=True)
        assert torch.equal(got.resolve_conj().resolve_neg(), table.resolve_conj().resolve_neg()[rows])


def test_found_values_under_vmap():
    m, q = _map()
    tables = torch.randn(3, 50, 2, device=DEV)

    def look(table):
        m.values["default"] = table
        return m.find(q, return_indices=False, return_values=True)[1]

    try:
        got = torch.func.vmap(look)(tables)
    finally:
        m.values["default"] = tables[0]
    _, rows = m.find(q)
    assert torch.equal(got, tables[:, rows])


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
