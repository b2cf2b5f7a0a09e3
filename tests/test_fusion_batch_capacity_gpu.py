"""Sequences into a map that runs full inside a batch, and into a bounded grid."""
import pytest
import torch

from test_fusion_batch_gpu import DEV, _content, _frames, _volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.5, 0.9])
@pytest.mark.parametrize("n,G", [(20, 8), (40, 8), (20, 5)])
def test_batch_into_a_full_map(n, G, share):
    """Which blocks get a row is open within a batch; each that has one holds what all frames give it, rows are handed out
    once, and threads that wait for a row which does not come end without a run-out wait."""
    import __ash
    from ash.fusion import TSDFFusion

    frames = _frames(n)
    ample = _volume(G, 5)
    TSDFFusion(ample, 1).fuse_dataset(frames)
    keys, values = _content(ample)
    capacity = int(share * len(keys))
    small = _volume(G, 5, capacity=capacity)
    TSDFFusion(small, 1).fuse_dataset(frames)
    assert small.engine.backend.status() == __ash.STATUS_CAPACITY
    got, rows = small.engine.items()
    assert len(got) == capacity == len(torch.unique(rows)) == len(torch.unique(got, dim=0))
    place = ample.engine.find(got.contiguous())
    assert place[1].all()
    assert torch.equal(small.embeddings.data[rows], ample.embeddings.data[place[0]])
    TSDFFusion(small, 1).fuse_dataset(frames)           # the blocks that are there are found again
    assert small.engine.backend.status() == __ash.STATUS_CAPACITY
    assert torch.equal(small.engine.items()[0].sort(dim=0)[0], got.sort(dim=0)[0])


def test_bounded_grid():
    """A sequence that leaves the box equals its frames, and no block outside the box comes to be."""
    import ash
    from ash.fusion import TSDFFusion

    frames, grids = _frames(35), []
    for whole in (True, False):
        grid = ash.BoundedSparseDenseGrid(3, 8000, 5, 8, 24, torch.full((3,), -1.2), torch.full((3,), 2.0), DEV)
        fusion = TSDFFusion(grid, 1)
        if whole:
            fusion.fuse_dataset(frames)
        else:
            for f in frames:
                fusion.fuse_frame(f)
        assert grid.engine.backend.status() == 0
        grids.append(grid)
    (ka, va), (kb, vb) = map(_content, grids)
    assert len(ka) > 50 and torch.equal(ka, kb) and torch.equal(va, vb) and (va[..., 4] > 0).any()
    assert (ka >= 0).all() and (ka < 24).all()
    free = _volume(8, 5, cell=grids[0].cell_size)
    TSDFFusion(free, 1).fuse_dataset(frames)
    assert free.engine.size() > len(ka)                 # the frames see more than the box holds
