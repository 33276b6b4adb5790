"""The gates of an mLSTM over whole sequences (64 rows and four heads at a time) against the same rows taken one by one: the same bits,
state included, at the edges of a chunk and of a group of heads, beside other sequences and rows of no sequence."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lens,slots", [([1], [0]), ([63, 64, 65], [2, 0, 1]), ([129, 7], [1, -1]), ([300], [0])])
@pytest.mark.parametrize("H", [1, 4, 5, 12])
@pytest.mark.parametrize("dtype,bad", [(torch.float32, False), (torch.bfloat16, False), (torch.float32, True)])
def test_whole_sequences_as_single_rows(lens, slots, H, dtype, bad):
    torch.manual_seed(H + sum(lens))
    T, off = sum(lens), 8
    pre, bias = 6 * torch.randn((T, 2 * H), device=DEV), torch.randn(2 * H, device=DEV).to(dtype)
    pre[T // 2, 0] = -1e4                                            # saturated gates
    pre[T // 3, H] = 1e4
    if bad:                                                          # both gates of the last row: m is not a number after it
        pre[-1, :] = float("nan")
    row0 = [sum(lens[:i]) for i in range(len(lens))]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    start = torch.randn((3, off + H), device=DEV)
    whole, one = start.clone(), start.clone()
    got = ops.mlstm_gates(pre, bias, 15.0, i32(row0), i32(lens), i32(slots), whole, off, len(lens), H)
    for r0, n, s in zip(row0, lens, slots):
        for t in range(r0, r0 + n):
            want = ops.mlstm_gates(pre[t:t + 1], bias, 15.0, None, None, i32([s]), one, off, 1, H)
            assert torch.equal(got[t:t + 1].view(torch.int32), want.view(torch.int32)), (t, s)
    assert torch.equal(whole.view(torch.int32), one.view(torch.int32))


def test_more_sequences_than_a_grid_has_rows():
    """65537 sequences of one row with their lengths given, as the same rows without."""
    n, i32 = 65537, lambda x: x.to(torch.int32)  # noqa: E731
    torch.manual_seed(1)
    pre, bias, start = torch.randn((n, 2), device=DEV), torch.randn(2, device=DEV), torch.randn((n, 1), device=DEV)
    at, ones = i32(torch.arange(n, device=DEV)), i32(torch.ones(n, device=DEV))
    whole, one = start.clone(), start.clone()
    got = ops.mlstm_gates(pre, bias, 15.0, at, ones, at, whole, 0, n, 1)
    assert torch.equal(got, ops.mlstm_gates(pre, bias, 15.0, None, None, at, one, 0, n, 1)) and torch.equal(whole, one)
