"""Batches of a sequence stand on their own: a word of frames that one leaves behind, as a pass whose copies ran out would,
does not keep its block out of the next."""
import pytest
import torch

from test_fusion_batch_gpu import DEV, _frames, _volume

pytestmark = pytest.mark.gpu


def test_a_word_left_behind():
    """The counter of fused blocks is laid over the word of a row that the second batch allocates, so that word is not zero
    when the batch begins.  Each batch is one view 32 times: whatever the counter adds to the word on the way, the
    frames that it names are the batch's own."""
    from ash.fusion import TSDFFusion

    first, second = _frames(1)[0], None
    for f in _frames(12):
        a, b = _volume(8, 5, capacity=4000), _volume(8, 5, capacity=4000)
        TSDFFusion(a, 1).fuse_frame(first), TSDFFusion(b, 1).fuse_dataset([first, f])
        if b.engine.size() - a.engine.size() > 20:      # a view with blocks of its own
            second = f
            break
    assert second is not None
    n_first, n_both = a.engine.size(), b.engine.size()
    for row in range(n_first + n_first % 2, n_both, 2):     # of even number: the counter's words have 64 bits
        grid = _volume(8, 5, capacity=4000)
        fusion = TSDFFusion(grid, 1)
        fusion._list2 = torch.zeros(2 * grid.num_embeddings + 1, dtype=torch.int32, device=DEV)
        word = fusion._list2[grid.num_embeddings:-1].view(torch.int64)[row // 2:row // 2 + 1]
        fusion.fuse_dataset([first] * 32 + [second] * 32, counter=word)
        keys, rows = grid.engine.items()
        assert len(keys) == n_both
        expected, b_rows = b.engine.items()
        want = b.embeddings.data[b_rows[(expected == keys[rows == row]).all(dim=1)]]
        if (want[..., 4] > 0).any():                        # the view observes the block that came to lie there
            assert (grid.embeddings.data[row, :, 4] > 0).any()
            return
    raise AssertionError("the second view observes none of its blocks")
