"""The separable window filter at every compiled-in block edge, radius and channel grouping, and beside them."""
import numpy as np
import pytest
import torch

import ash

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("G", [4, 8, 16, 5])
@pytest.mark.parametrize("R", [1, 2, 3])
@pytest.mark.parametrize("D", [1, 2, 4, 6, 8, 13])
def test_separable_filter_equals_float64_window(G, R, D):
    """Three factors per channel against the same three sums taken in float64 over the dense volume that the
    blocks fill.  Each sum of S = 2R + 1 products in float32 is off by at most S 2^-24 of the sum of the terms'
    magnitudes, three passes by 3 S 2^-24 of the magnitudes filtered with |w|."""
    import __ash as native

    S, n = 2 * R + 1, 11
    g = torch.Generator(device=DEV).manual_seed(100 * G + 10 * R + D)
    cells = torch.randperm(27, generator=g, device=DEV)[:n]     # 11 of the 27 blocks of a cube: many neighbours absent
    coords = torch.stack([cells % 3, cells // 3 % 3, cells // 9], 1).int()
    grid = ash.SparseDenseGrid(3, n + 4, D, G, DEV)
    grid.engine.insert_keys(coords)
    x = torch.randn(n + 4, G**3, D, generator=g, device=DEV)
    w = torch.randn(3, S, D, generator=g, device=DEV)
    _, lut = grid.construct_grid_neighbor_lut(1, bidirectional=True)
    keys, index = grid.engine.items()
    got = native.convolution_forward_separable(x, w, index.view(-1, 1), lut, G, R)

    def filtered(values, weights):
        v = torch.zeros(5 * G, 5 * G, 5 * G, D, dtype=torch.float64, device=DEV)     # z, y, x; a block of zeros all around
        at = [slice(int(c) * G + G, int(c) * G + 2 * G) for c in keys.flatten().tolist()]
        for i, b in enumerate(index.tolist()):
            v[at[3 * i + 2], at[3 * i + 1], at[3 * i]] = values[b].view(G, G, G, D).double()
        for axis, factor in zip((2, 1, 0), weights.double()):
            v = sum(torch.roll(v, R - k, dims=axis) * factor[k] for k in range(S))
        return torch.stack([v[at[3 * i + 2], at[3 * i + 1], at[3 * i]].reshape(G**3, D) for i in range(n)])

    bound = 3 * S * 2.0**-24 * filtered(x.abs(), w.abs())
    assert ((got[index].double() - filtered(x, w)).abs() <= bound + 1e-30).all()
    spare = np.setdiff1d(np.arange(n + 4), index.cpu().numpy())
    assert got[torch.from_numpy(spare).to(DEV)].abs().max() == 0
