"""The native pass over padded host batches against the tensor operations it stands for."""
import numpy as np
import pytest
import torch

from supertoken_b200.bpe_trainer import _flatten_batch, _flatten_batches


@pytest.mark.parametrize("top,marks", [(256, torch.uint8), (257, torch.bool), (70000, torch.uint8)])
def test_padded_batches_flatten_alike(top, marks):
    g = torch.Generator().manual_seed(top)
    batches = []
    for rows, width in ((3, 7), (16, 200), (1, 1), (0, 5), (5, 0)):
        lengths = torch.randint(0, width + 1, (rows, 1), generator=g)
        valid = torch.arange(width)[None, :] < lengths
        batches.append((torch.randint(0, top, (rows, width), generator=g, dtype=torch.int32), valid.to(marks)))
    ref = [_flatten_batch(b) for b in batches]
    (ids, off), = _flatten_batches(batches)
    assert ids.dtype == (torch.uint8 if top <= 256 else torch.int32)
    assert torch.equal(ids.to(torch.int32), torch.cat([i for i, _ in ref]))
    assert np.array_equal(np.diff(off), np.concatenate([np.diff(o) for _, o in ref]))
    batches[1][1][2] = torch.tensor([1, 0] * 100).to(marks)
    with pytest.raises(ValueError):
        _flatten_batches(batches)
    wide = [(b[0].to(torch.int64), b[1]) for b in batches[:1]]  # another type: the tensor operations
    assert torch.equal(_flatten_batches(wide)[0][0], ref[0][0])
