"""Indices of the row list where one lane writes all eight pairs of a query: two at a time where the list starts on 16 bytes,
one at a time where it does not, the same either way."""
import pytest
import torch

from test_fused_gpu import DEV, _make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("second", [False, True])
@pytest.mark.parametrize("dtype,D", [(torch.float32, 1), (torch.float32, 2), (torch.float32, 4), (torch.float32, 3),
                                     (torch.float64, 1), (torch.float64, 2)])
def test_lists_of_both_alignments(dtype, D, second):
    import __ash

    grid, x = _make("unbounded", 4, D, seed=29)
    x = x[:1003].contiguous()
    emb, n = grid.embeddings.detach().to(dtype), x.shape[0]
    origin, cell_size = grid._cell_frame()
    hm, lut = grid.engine.backend, grid._neighbor_lut32()
    g = torch.Generator(device=DEV).manual_seed(D)
    z = torch.randn(n, D, generator=g, device=DEV, dtype=dtype)
    ggx = torch.randn(n, 3, generator=g, device=DEV, dtype=dtype) if second else None
    _, masks, bidx = __ash.grid_query_forward(hm, emb, x, cell_size, origin, 4, lut, "linear")
    assert 0.2 < float(masks.float().mean()) < 0.95
    idx, rows, side = __ash.grid_query_backward_rows(hm, z, emb, x, cell_size, origin, 4, lut, bidx, "linear", grad_grad_x=ggx)
    assert idx.data_ptr() % 16 == 0
    off = torch.full((16 * n + 2,), -7, dtype=torch.int64, device=DEV)
    off_rows, off_side = torch.empty_like(rows), torch.empty_like(side)
    __ash._check(__ash._lib.ashb_grid_query_backward_rows(
        hm._h, __ash._dtype_code(emb), __ash._interp_code("linear"), int(second), ggx.data_ptr() if second else None, z.data_ptr(),
        emb.data_ptr(), x.data_ptr(), float(cell_size), __ash._host_floats(origin, 3), 4, lut.data_ptr(), bidx.data_ptr(),
        off[1:].data_ptr(), off_rows.data_ptr(), off_side.data_ptr(), n, emb.shape[0], D, __ash._stream(emb.device)))
    assert torch.equal(off[1:-1].view(2, -1), idx) and off[0] == -7 and off[-1] == -7
    assert torch.equal(off_rows, rows) and torch.equal(off_side, side)
    assert (idx >= 0).all() and (idx[0] < emb.shape[0]).all() and (idx[1] < 64).all()
    reached = torch.zeros_like(emb)
    __ash.rows_scatter_add(reached, idx, rows)
    if not second:      # up to 8 n terms, in any order
        dense = __ash.grid_query_backward(hm, z, emb, x, cell_size, origin, 4, lut, bidx, "linear")[0]
        torch.testing.assert_close(reached, dense, rtol=2e-5, atol=2e-5 * float(dense.abs().max()))
