"""A sequence of frames is fused in batches, one pass over the blocks for all frames of a batch, and the means of a cell
share one reciprocal: the volume equals, bit for bit, the one that single frames and IEEE divisions give."""
import numpy as np
import pytest
import torch

import bench_workloads as bw

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _frames(n, H=48, W=64, tilt=0.0):
    import ash

    scene, K = bw.Scene(DEV), bw.intrinsics(H, W)
    K_used = K.clone()
    K_used[2, 0] = tilt      # not the usual matrix: its last row is multiplied out
    frames = []
    for pose in bw.camera_poses(n, seed=5):
        depth, color = scene.render(K.to(DEV), pose.float().to(DEV), H, W)
        frames.append(ash.DotDict(depth=depth, depth_scale=1.0, depth_max=5.0, intrinsic=K_used,
                                  extrinsic=torch.linalg.inv(pose), rgb=color))
    return frames


def _volume(G, D, capacity=40_000, cell=0.04):
    import ash

    grid = ash.UnBoundedSparseDenseGrid(3, capacity, D, G, cell_size=cell * 8 / G, device=DEV)
    return grid


def _content(grid):
    keys, rows = grid.engine.items()
    order = torch.from_numpy(np.lexsort(keys.cpu().numpy().T[::-1])).to(DEV)
    return keys[order], grid.embeddings.data[rows[order]]


# one frame more than a batch, two batches, a single pair; rows that travel by bulk copies and rows that do not (G = 5, 3)
@pytest.mark.parametrize("n,G,D,tilt", [(2, 8, 5, 0.0), (32, 8, 5, 0.0), (33, 8, 6, 0.0), (64, 4, 5, 0.0), (35, 5, 5, 0.0),
                                         (5, 16, 5, 0.0), (3, 3, 7, 0.0), (40, 8, 5, 0.01), (40, 5, 5, 0.01)])
def test_sequence_equals_its_frames(n, G, D, tilt):
    from ash.fusion import TSDFFusion

    frames = _frames(n, tilt=tilt)
    a, b = _volume(G, D), _volume(G, D)
    counters = [torch.zeros(1, dtype=torch.int64, device=DEV) for _ in range(2)]
    whole, single = TSDFFusion(a, 1), TSDFFusion(b, 1)
    whole.fuse_dataset(frames, counter=counters[0])
    for f in frames:
        single.fuse_frame(f, counter=counters[1])
    (ka, va), (kb, vb) = _content(a), _content(b)
    assert len(ka) > 50 and torch.equal(ka, kb) and torch.equal(va, vb) and (va[..., 4] > 0).any()
    assert int(counters[0]) == int(counters[1])
    whole.fuse_frame(frames[0]), single.fuse_frame(frames[0])     # the stamps go on where the sequence ended
    assert torch.equal(_content(a)[1], _content(b)[1])
    whole.fuse_dataset(frames[:2]), single.fuse_dataset(frames[:1]), single.fuse_dataset(frames[1:2])
    assert torch.equal(_content(a)[1], _content(b)[1])
    assert a.engine.backend.status() == 0 and b.engine.backend.status() == 0


@pytest.mark.parametrize("G", [8, 5])
def test_divisions_of_extreme_values(G):
    """Means and weights from the whole range of floats: zeros of both signs, denormals, infinities, NaN, divisors beyond
    what shares a reciprocal."""
    from ash.fusion import TSDFFusion
    from oracle import tsdf as otsdf

    (f,), cell = _frames(1), 0.04 * 8 / G
    grid = _volume(G, 5, capacity=6000)
    fusion, ref = TSDFFusion(grid, 1), otsdf.OracleTSDF(6000, G, cell, 1)
    E = f.extrinsic.numpy()
    observe = lambda: ref.fuse_frame(f.depth.cpu().numpy(), f.rgb.cpu().numpy(), f.intrinsic.numpy(), E, np.linalg.inv(E), 5.0)
    fusion.fuse_frame(f), observe()
    keys, rows = grid.engine.items()
    rk, ridx = ref.map.items()
    order, rorder = np.lexsort(keys.cpu().numpy().T[::-1]), np.lexsort(rk.T[::-1])
    rng = np.random.default_rng(G)
    shape = (len(rk), G**3, 5)
    values = np.where(rng.random(shape) < 0.5, rng.integers(0, 2**32, shape, dtype=np.uint32).view(np.float32),
                      rng.standard_normal(shape).astype(np.float32) * np.float32(10.0) ** rng.integers(-6, 7, shape)).astype(np.float32)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, -1e-45, 3.4e38, 2.0**90, 2.0**-90], np.float32)
    values = np.where(rng.random(shape) < 0.1, rng.choice(special, shape), values)
    values[..., 4] = np.where(rng.random(shape[:2]) < 0.8, np.abs(rng.integers(0, 500, shape[:2])), values[..., 4])
    ref.emb[ridx[rorder]] = values
    grid.embeddings.data[rows[torch.from_numpy(order).to(DEV)]] = torch.from_numpy(values).to(DEV)
    with np.errstate(all="ignore"):
        fusion.fuse_frame(f), observe()
    got = grid.embeddings.data[rows[torch.from_numpy(order).to(DEV)]].cpu().numpy()
    np.testing.assert_array_equal(got, ref.emb[ridx[rorder]])
