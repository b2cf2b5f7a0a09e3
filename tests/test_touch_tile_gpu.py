"""Block allocation drops repeated blocks within a tile of 512 points.  The blocks it allocates, against the
numpy restatement, where the tile is ragged, its set of seen blocks overflows, or its blocks lie further
apart than the set can tell."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _blocks(grid):
    c = grid.engine.items()[0].cpu().numpy()
    return c[np.lexsort(c.T[::-1])]


@pytest.mark.parametrize("n,spread,dilation", [(1, 1.0, 1), (511, 0.5, 1), (513, 40.0, 0), (700, 3000.0, 1), (1500, 8.0, 2),
                                               (300, 500.0, 4)])
def test_points(n, spread, dilation):
    import ash
    from oracle.tsdf import touched_blocks

    g = torch.Generator(device=DEV).manual_seed(n)
    pts = (torch.rand(n, 3, generator=g, device=DEV) - 0.5) * spread
    pts[: n // 3] = pts[n // 3: 2 * (n // 3)]                                # repeats in other warps and tiles
    ref = touched_blocks(pts.cpu().numpy(), 0.05, [0, 0, 0], 8, dilation)
    grid = ash.UnBoundedSparseDenseGrid(3, len(ref), 1, 8, cell_size=0.05, device=DEV)
    grid.spatial_init_(pts, dilation=dilation, bidirectional=True)
    np.testing.assert_array_equal(_blocks(grid), ref)


@pytest.mark.parametrize("H,W,step,dilation", [(1, 1, 0.0, 1), (17, 33, 0.3, 1), (64, 31, 90.0, 1), (15, 640, 0.01, 2)])
def test_frames(H, W, step, dilation):
    import ash
    from ash.fusion import TSDFFusion
    from oracle.tsdf import touched_blocks, unproject

    g = torch.Generator(device=DEV).manual_seed(H)
    depth = 1.0 + step * torch.randint(0, 20, (H, W), generator=g, device=DEV)
    depth[torch.rand(H, W, generator=g, device=DEV) < 0.1] = 0.0
    depth[0, 0] = 1.5
    K = np.array([[W, 0, W / 2], [0, W, H / 2], [0, 0, 1.0]], dtype=np.float32)
    ref = touched_blocks(unproject(depth.cpu().numpy(), K, np.eye(4), 3000.0), 0.02, [0, 0, 0], 8, dilation)
    grid = ash.UnBoundedSparseDenseGrid(3, len(ref), 5, 8, cell_size=0.02, device=DEV)
    TSDFFusion(grid, dilation).fuse_frame(ash.DotDict(
        depth=depth, depth_scale=1.0, depth_max=3000.0, intrinsic=K, extrinsic=np.eye(4), rgb=torch.rand(H, W, 3, device=DEV)))
    np.testing.assert_array_equal(_blocks(grid), ref)


@pytest.mark.parametrize("n,dilation", [(5_000, 2), (60_000, 2), (150_000, 1), (300_000, 1)])
def test_scattered_points(n, dilation):
    """A block each: the neighbours of 512 points are shared out among eight, four, two and one CTA."""
    import ash
    from oracle.tsdf import touched_blocks

    g = torch.Generator(device=DEV).manual_seed(n)
    pts = torch.rand(n, 3, generator=g, device=DEV) - 0.5
    ref = touched_blocks(pts.cpu().numpy(), 0.01, [0, 0, 0], 8, dilation)
    grid = ash.UnBoundedSparseDenseGrid(3, len(ref), 1, 8, cell_size=0.01, device=DEV)
    coords, _, index, _ = grid.spatial_init_(pts, dilation=dilation, bidirectional=True)
    np.testing.assert_array_equal(_blocks(grid), ref)
    assert torch.equal(torch.sort(index.view(-1)).values, torch.arange(len(ref), device=DEV))
    assert torch.equal(grid.engine.find(coords.view(-1, 3))[0], index.view(-1))
