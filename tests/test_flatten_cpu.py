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


def _refilled(batches):
    """What a loader with one buffer yields: views of it, refilled for every batch."""
    cells = max(b[0].numel() for b in batches)
    tokens, valid = torch.empty(cells, dtype=torch.int32), torch.empty(cells, dtype=batches[0][1].dtype)
    for t, v in batches:
        tokens.fill_(77), valid.fill_(1)
        tokens[:t.numel()], valid[:t.numel()] = t.reshape(-1), v.reshape(-1)
        yield tokens[:t.numel()].reshape(t.shape), valid[:t.numel()].reshape(t.shape), None
    tokens.fill_(88), valid.fill_(1)


@pytest.mark.parametrize("tops", [(256,) * 40, (256, 256, 300) + (200,) * 30, (70000, 5), (9,)])
@pytest.mark.parametrize("shapes", [((2, 3),), ((0, 4), (5, 0), (1, 1), (8, 100)), ((64, 31), (3, 2))])
def test_batches_of_a_loader_that_refills_its_buffers(tops, shapes):
    # ids from 256 on in some later batch, growth beyond the first batch's room, empty batches first
    g = torch.Generator().manual_seed(len(tops))
    batches = []
    for i, top in enumerate(tops):
        rows, width = shapes[i % len(shapes)]
        valid = (torch.arange(width)[None, :] < torch.randint(0, width + 1, (rows, 1), generator=g)).to(torch.uint8)
        batches.append((torch.randint(0, top, (rows, width), generator=g, dtype=torch.int32), valid))
    ref = [_flatten_batch(b) for b in batches]
    (ids, off), = _flatten_batches(_refilled(batches))
    assert torch.equal(ids.to(torch.int32), torch.cat([i for i, _ in ref]))
    assert off[0] == 0 and np.array_equal(np.diff(off), np.concatenate([np.diff(o) for _, o in ref]))
