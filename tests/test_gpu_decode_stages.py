"""Decode attention at head size 256 with more blocks than the device holds with three stages, several hundred keys in every range, so that
the two-stage ring is refilled: one range, ranges merged in clusters or by the combine kernel, odd tails, a window, a wrapped ring."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE, NQ, NKV, HD = 64, 8, 4, 256


def batch(B, ring, seed):
    """Rows, pools, page tables and lengths of B sequences of 300 to 1200 tokens, and their keys and values in order of position."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    lens = [300 + (b * 97 + seed) % 900 for b in range(B)]
    per = (ring or 1216) // PAGE
    keys, values = (torch.randn((B, 1216, NKV, HD), device=DEV, generator=g).bfloat16() for _ in range(2))
    table = (torch.randperm(B * per, device=DEV, generator=g).to(torch.int32) + 1).view(B, per)
    pools = torch.zeros((2, B * per + 1, NKV, PAGE, HD), dtype=torch.bfloat16, device=DEV)
    for b, n in enumerate(lens):
        pos = torch.arange(max(0, n - ring) if ring else 0, n, device=DEV)
        cell = pos % ring if ring else pos
        pages = table[b].long()[cell // PAGE]
        pools[0, pages, :, cell % PAGE] = keys[b, pos]
        pools[1, pages, :, cell % PAGE] = values[b, pos]
    qkv = torch.randn((B, (NQ + 2 * NKV) * HD), device=DEV, generator=g).bfloat16()
    return lens, table, pools, qkv, keys, values


def decode(rows, lens, table, pools, qkv, splits, window, cap, ring, uneven):
    B = len(rows)
    part_o, part_ml = torch.empty(B * NQ * splits * HD, device=DEV), torch.empty(B * NQ * splits * 2, device=DEV)
    slot_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    return ops.attn_decode(qkv[rows].contiguous(), NQ, NKV, HD, pools[0], pools[1], table, PAGE, ring, torch.tensor(rows, dtype=torch.int32, device=DEV),
                           slot_len, HD ** -0.5, cap, window, splits, part_o, part_ml, uneven=uneven)


def exact(b, n, qkv, keys, values, window, cap):
    lo = max(0, n - window) if window else 0
    q = qkv[b, :NQ * HD].double().view(NKV, NQ // NKV, HD)
    s = torch.einsum("khd,pkd->khp", q, keys[b, lo:n].double()) * HD ** -0.5
    p = (cap * torch.tanh(s / cap) if cap else s).softmax(-1)
    return torch.einsum("khp,pkd->khd", p, values[b, lo:n].double()).reshape(-1)


@pytest.mark.parametrize("splits,B", [(1, 75), (1, 120), (2, 38), (3, 25), (4, 19), (4, 40), (6, 13), (6, 20)])
@pytest.mark.parametrize("window,cap,ring", [(None, 50.0, 0), (None, None, 0), (333, None, 0), (512, 50.0, 512)])
def test_two_stages(splits, B, window, cap, ring):
    lens, table, pools, qkv, keys, values = batch(B, ring, splits + B)
    every = list(range(B))
    got = decode(every, lens, table, pools, qkv, splits, window, cap, ring, True)
    for b in every[::max(1, B // 16)]:
        want = exact(b, lens[b], qkv, keys, values, window, cap)
        # bfloat16 weights beside float32 sums, and the result's own rounding
        assert ((got[b].double() - want).norm() / want.norm()).item() < 8e-3, b
    few = max(1, 296 // (NKV * splits))                          # blocks that fit at once: three stages
    parts = torch.cat([decode(every[lo:lo + few], lens, table, pools, qkv, splits, window, cap, ring, True) for lo in range(0, B, few)])
    assert ((got.double() - parts.double()).norm() / parts.double().norm()).item() < 4e-3       # a rounding of the result, where the merge differs
    if splits > 4:
        assert torch.equal(got, parts)                           # the combine kernel either way, so the ranges' own sums are the same
    other = decode(every, lens, table, pools, qkv, splits, window, cap, ring, False)
    assert ((got.double() - other.double()).norm() / other.double().norm()).item() < 4e-3
