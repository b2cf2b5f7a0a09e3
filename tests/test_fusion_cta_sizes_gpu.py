"""The fusion pass takes more threads a CTA where a block's rows leave an SM room for few CTAs: single frames and a sequence
against the restatement, at block edges and channel counts on both sides of each line."""
import numpy as np
import pytest
import torch

from test_fusion_batch_gpu import DEV, _content, _frames, _volume

pytestmark = pytest.mark.gpu


# bytes of the tiles of a CTA: 20 KB (128 threads), 33 to 39 KB and 55 KB (256, an odd count of CTAs too), 80 KB and up (512)
@pytest.mark.parametrize("G,D", [(8, 5), (8, 9), (8, 10), (8, 16), (9, 5), (10, 5), (12, 5), (14, 5), (15, 5), (16, 5), (16, 12),
                                 (5, 16)])
@pytest.mark.parametrize("tilt", [0.0, 0.01])
def test_frames_equal_the_restatement(G, D, tilt):
    _compare(G, D, tilt, 0.04)


# cells two pixels apart and more at the largest depth: a single frame of block edge 8 takes 256 threads
@pytest.mark.parametrize("G,D,cell", [(8, 5, 0.18), (8, 5, 0.2), (8, 9, 0.2), (8, 16, 0.2), (4, 5, 0.2), (5, 5, 0.2)])
def test_coarse_cells(G, D, cell):
    _compare(G, D, 0.0, cell)


def _compare(G, D, tilt, cell):
    from ash.fusion import TSDFFusion
    from oracle import tsdf as otsdf

    frames = _frames(3, tilt=tilt)
    grids = [_volume(G, D, capacity=4000, cell=cell) for _ in range(2)]
    ref = otsdf.OracleTSDF(4000, G, grids[0].cell_size, 1)
    single, whole = (TSDFFusion(g, 1) for g in grids)
    whole.fuse_dataset(frames)
    for f in frames:
        E = f.extrinsic.numpy()
        single.fuse_frame(f)
        ref.fuse_frame(f.depth.cpu().numpy(), f.rgb.cpu().numpy(), f.intrinsic.numpy(), E, np.linalg.inv(E), 5.0)
    rk, ridx = ref.map.items()
    rorder = np.lexsort(rk.T[::-1])
    for g in grids:
        keys, values = _content(g)
        np.testing.assert_array_equal(keys.cpu().numpy(), rk[rorder])
        np.testing.assert_array_equal(values[..., :5].cpu().numpy(), ref.emb[ridx[rorder]])
        assert (values[..., 4] > 0).any() and not values[..., 5:].any()
        assert g.engine.backend.status() == 0
