"""Prompt attention with a running maximum: two groups of warps share a row's maximum, so rows whose maximum lies in either group's
tiles, grows late, or is missing from a whole tile (a window's edge, a row's last key) have to come out as float64 gives them."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def exact(qkv, lens, nq, nkv, hd, window, slopes):
    out, r0 = [], 0
    for n in lens:
        x = qkv[r0:r0 + n].double().view(n, nq + 2 * nkv, hd).transpose(0, 1)
        q, k, v = x[:nq], x[nq:nq + nkv].repeat_interleave(nq // nkv, 0), x[nq + nkv:].repeat_interleave(nq // nkv, 0)
        i = torch.arange(n, device=DEV)
        d = i[:, None] - i[None, :]
        s = q @ k.transpose(1, 2) * hd ** -0.5
        if slopes is not None:
            s = s - slopes.double()[:, None, None] * d
        s = s.masked_fill((d < 0) | (d >= (window or n)), float("-inf"))
        out.append((s.softmax(-1) @ v).transpose(0, 1).reshape(n, nq * hd))
        r0 += n
    return torch.cat(out)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("lens", [[1], [64], [65, 128, 129, 1], [700], [1024]])
@pytest.mark.parametrize("window,slope,grow", [(None, None, 0.0), (1, None, 0.0), (65, None, 0.0), (100, 0.5, 0.0), (None, None, 30.0), (None, None, -30.0)])
def test_running_maximum(hd, lens, window, slope, grow):
    nq, nkv, T = 4, 2, sum(lens)
    torch.manual_seed(hd + T)
    qkv = torch.randn((T, nq + 2 * nkv, hd), device=DEV)
    if grow:                                         # one direction that keys go along more and more (or less and less)
        at = torch.cat([torch.linspace(0, 1, n) for n in lens]).to(DEV)
        qkv[:, :nq, 0] = abs(grow)
        qkv[:, nq:nq + nkv, 0] = (at * grow)[:, None]
    qkv = qkv.reshape(T, -1).bfloat16()
    row0 = torch.tensor([sum(lens[:i]) for i in range(len(lens))], dtype=torch.int32, device=DEV)
    ln = torch.tensor(lens, dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n) for n in lens]).to(DEV, torch.int32)
    slopes = None if slope is None else torch.linspace(0.0, slope, nq, device=DEV)
    got = ops.attn_prefill(qkv, nq, nkv, hd, pos, row0.repeat_interleave(ln), hd ** -0.5, None, window, row0, ln, max(lens), slopes=slopes)
    ops.raise_on_status(torch.device(DEV))
    want = exact(qkv, lens, nq, nkv, hd, window, slopes)
    # weights and results are rounded to bfloat16: two roundings of 2^-9 relative, in root mean square less
    assert ((got.double() - want).norm() / want.norm()).item() < 2.0 ** -8
    assert (got.double() - want).abs().max().item() < 2.0 ** -6 * max(1.0, want.abs().max().item())
