"""The ring of pinned buffers: arrays of one byte to more than a buffer, more of them than buffers, sent without waiting."""
import numpy as np
import pytest
import torch

from quicknn_b200.cache.upload import PinnedUploader

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries,nbytes", [(1, 16), (3, 64), (8, 1 << 16)])
def test_ring(entries, nbytes):
    up, rng, sent = PinnedUploader("cuda:0", entries, nbytes), np.random.default_rng(1), []
    for i in range(4 * entries + 3):
        a = rng.integers(0, 256, [1, nbytes, nbytes + 1, 3, 5 * nbytes][i % 5], dtype=np.uint8)
        t = torch.empty(a.size, dtype=torch.uint8, device="cuda:0")
        up.send(t, a)
        sent.append((t, a.copy()))
        a[:] = 0                                                    # the caller's array is its own again at once
    assert all((t.cpu().numpy() == a).all() for t, a in sent)
    up.send(torch.empty(0, dtype=torch.int32, device="cuda:0"), np.zeros(0, np.int32))
    with pytest.raises(ValueError):
        up.send(torch.empty(2, dtype=torch.int32, device="cuda:0"), np.zeros(3, np.int32))
