"""The ring of pinned buffers: arrays of one byte to more than a buffer, more of them than buffers, sent without waiting."""
import threading

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


def test_host_memory_and_threads():
    """A destination in host memory has its bytes at once; threads that share a ring get their own."""
    up = PinnedUploader("cuda:0", 2, 4096)
    t = torch.empty(3, dtype=torch.int32)
    up.send(t, np.array([5, 6, 7], np.int32))
    assert t.tolist() == [5, 6, 7]
    rng = np.random.default_rng(2)
    data = rng.integers(0, 256, (4, 200, 4096), dtype=np.uint8)
    out = torch.zeros((4, 200, 4096), dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()

    def work(i):
        for j in range(200):
            up.send(out[i, j], data[i, j])
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert (out.cpu().numpy() == data).all()
