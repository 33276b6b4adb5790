"""Steps that continue sequences, over the pages of the cache: the bits of the same step over packed copies of the sequences, wherever
the new rows begin in a page or a tile, beside fresh sequences, under a window, in pairs of CTAs, and with Inf and NaN left in cells
behind a sequence."""
from types import SimpleNamespace

import pytest
import torch

from quicknn_b200.engine.batch import WholeSequences
from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("starts,news", [([1], [1]), ([64], [64]), ([63, 0, 128], [2, 65, 1]), ([100, 1000, 0, 777], [28, 203, 300, 129]),
                                         ([2900], [130]), ([127, 500, 64], [129, 12, 500])])
@pytest.mark.parametrize("cap,window,slopes", [(50.0, None, False), (None, None, False), (50.0, 90, False), (None, 300, True)])
def test_same_bits_as_packed_rows(hd, starts, news, cap, window, slopes):
    nq, nkv, B = 4, 2, len(starts)
    torch.manual_seed(hd + sum(starts) + sum(news))
    lens = [s + n for s, n in zip(starts, news)]
    per, T = max((n + PAGE - 1) // PAGE for n in lens) + 1, sum(news)
    pages = B * per + 1
    pool = torch.randn((2, pages, nkv, PAGE, hd), device=DEV).bfloat16()
    table = (torch.randperm(pages - 1, device=DEV)[:B * per].to(torch.int32) + 1).view(B, per).contiguous()
    for b, n in enumerate(lens):                              # what earlier sequences may have left behind this one's
        page = int(table[b, (n - 1) // PAGE])
        pool[:, page, :, (n - 1) % PAGE + 1:] = float("nan") if b % 2 else float("inf")
    order = torch.randperm(B).tolist()                         # slots in another order than the step's
    slots = i32(order)
    slot_len, tab = torch.zeros(B, dtype=torch.int32, device=DEV), torch.empty_like(table)
    for b, s in enumerate(order):
        slot_len[s], tab[s] = lens[b], table[b]
    qkv = torch.randn((T, (nq + 2 * nkv) * hd), device=DEV).bfloat16()
    new0, row0 = [sum(news[:i]) for i in range(B)], [sum(lens[:i]) for i in range(B)]
    pos = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, news)]).to(DEV, torch.int32)
    ln = i32(news)
    whole = WholeSequences(slots, i32(starts), i32(new0), ln, i32(row0), i32(lens), i32(row0).repeat_interleave(ln) + pos, total=sum(lens),
                           longest=max(lens), most_new=max(news))
    line = SimpleNamespace(k=pool[0], v=pool[1], page_table=tab, page_size=PAGE, ring=0, slot_len=slot_len, writes=True, has_values=True)
    tok_slot = slots.repeat_interleave(ln)
    sl = torch.linspace(0.01, 0.4, nq, device=DEV) if slopes else None
    want = ops.attn_extend(qkv, nq, nkv, hd, line.k, line.v, tab, PAGE, 0, pos, i32(new0).repeat_interleave(ln), tok_slot, hd ** -0.5, cap, window,
                           whole=whole, slopes=sl)
    ops.cache_append(qkv, nq, nkv, hd, pos, tok_slot, line)
    assert ops.extends_in_pages(qkv, hd, line, whole)
    got = ops.attn_extend_paged(qkv, nq, nkv, hd, line, hd ** -0.5, cap, window, whole, slopes=sl)
    ops.raise_on_status(torch.device(DEV))
    assert torch.isfinite(want.float()).all() and torch.equal(got, want)


def test_where_pages_do_not_serve():
    line = SimpleNamespace(k=torch.zeros((2, 1, 64, 64), dtype=torch.bfloat16, device=DEV), page_size=64, ring=0, writes=True, has_values=True)
    whole = SimpleNamespace(longest=129, most_new=5)
    x = torch.zeros((5, 192), dtype=torch.bfloat16, device=DEV)
    takes = lambda **kw: ops.extends_in_pages(x, kw.pop("hd", 64), SimpleNamespace(**{**vars(line), **kw}), whole)  # noqa: E731
    assert takes() and takes(ring=192)
    assert not takes(ring=128) and not takes(page_size=32) and not takes(writes=False) and not takes(has_values=False) and not takes(hd=96)
    assert not ops.extends_in_pages(x, 64, line, None) and not ops.extends_in_pages(x.float(), 64, line, whole)


def exact(q, keys, values, first, scale, cap, window, sinks):
    """Attention in 64 bits of rows at positions first .. over keys and values [positions, kv heads, size]."""
    nq, nkv = q.shape[1], keys.shape[1]
    k, v = (t.double().repeat_interleave(nq // nkv, 1) for t in (keys, values))
    s = torch.einsum("qhd,phd->hqp", q.double(), k) * scale
    s = cap * torch.tanh(s / cap) if cap else s
    pos, row = torch.arange(k.shape[0], device=DEV), first + torch.arange(q.shape[0], device=DEV)
    seen = pos[None, :] <= row[:, None]
    if window:
        seen &= pos[None, :] > row[:, None] - window
    s = s.masked_fill(~seen, float("-inf"))
    if sinks is not None:
        s = torch.cat([s, sinks.double()[:, None, None].expand(-1, s.shape[1], 1)], -1)
    return torch.einsum("hqp,phd->qhd", s.softmax(-1)[..., :k.shape[0]], v)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("cap", [None, 50.0])
@pytest.mark.parametrize("ring,window", [(0, None), (256, 200)])
@pytest.mark.parametrize("with_sinks", [False, True])
def test_against_64_bits_in_a_ring_that_is_just_full_and_with_sinks(hd, cap, ring, window, with_sinks):
    nq, nkv, starts, news = 4, 2, [100, 0, 63, 192], [156, 256, 65, 3]       # the longest: 256 positions
    torch.manual_seed(hd)
    lens, B, T = [s + n for s, n in zip(starts, news)], len(starts), sum(news)
    per = 4
    pool = torch.full((2, B * per + 1, nkv, PAGE, hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    tab = (torch.randperm(B * per, device=DEV).to(torch.int32) + 1).view(B, per)
    new0, row0 = [sum(news[:i]) for i in range(B)], [sum(lens[:i]) for i in range(B)]
    ln = i32(news)
    pos = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, news)]).to(DEV, torch.int32)
    slots = i32(list(range(B)))
    tok_slot = slots.repeat_interleave(ln)
    whole = WholeSequences(slots, i32(starts), i32(new0), ln, i32(row0), i32(lens), i32(row0).repeat_interleave(ln) + pos, total=sum(lens),
                           longest=max(lens), most_new=max(news))
    line = SimpleNamespace(k=pool[0], v=pool[1], page_table=tab, page_size=PAGE, ring=ring, slot_len=i32(lens), writes=True, has_values=True)
    keys, values = (torch.randn((B, 256, nkv, hd), device=DEV).bfloat16() for _ in range(2))
    qkv = torch.randn((T, (nq + 2 * nkv) * hd), device=DEV).bfloat16()
    for b in range(B):
        p = torch.arange(starts[b], device=DEV)
        pages = tab[b].long()[p // PAGE]
        pool[0, pages, :, p % PAGE], pool[1, pages, :, p % PAGE] = keys[b, p], values[b, p]
        rows = qkv[new0[b]:new0[b] + news[b]]
        keys[b, starts[b]:lens[b]] = rows[:, nq * hd:(nq + nkv) * hd].reshape(-1, nkv, hd)
        values[b, starts[b]:lens[b]] = rows[:, (nq + nkv) * hd:].reshape(-1, nkv, hd)
    sinks = torch.randn(nq, device=DEV) if with_sinks else None
    want = ops.attn_extend(qkv, nq, nkv, hd, line.k, line.v, tab, PAGE, ring, pos, i32(new0).repeat_interleave(ln), tok_slot, hd ** -0.5, cap, window,
                           whole=whole, sinks=sinks)
    ops.cache_append(qkv, nq, nkv, hd, pos, tok_slot, line)
    assert ops.extends_in_pages(qkv, hd, line, whole)
    got = ops.attn_extend_paged(qkv, nq, nkv, hd, line, hd ** -0.5, cap, window, whole, sinks=sinks)
    ops.raise_on_status(torch.device(DEV))
    assert torch.equal(got, want)
    for b in range(B):
        rows = slice(new0[b], new0[b] + news[b])
        ref = exact(qkv[rows, :nq * hd].reshape(-1, nq, hd), keys[b, :lens[b]], values[b, :lens[b]], starts[b], hd ** -0.5, cap, window, sinks)
        assert ((got[rows].double() - ref.reshape(news[b], -1)).norm() / ref.norm()).item() < 8e-3, b       # bfloat16 weights and result
    # the cells behind a sequence in its last page are zero, those in front of them as they were
    for b, n in enumerate(lens):
        page = int(tab[b, (n - 1) // PAGE])
        assert (pool[1, page, :, (n - 1) % PAGE + 1:] == 0).all() and torch.equal(pool[1, page, :, (n - 1) % PAGE], values[b, n - 1])


def test_rows_that_the_kernel_does_not_take_go_the_general_way():
    """What the launcher would refuse (rows off 16 bytes) is not taken by the predicate."""
    line = SimpleNamespace(k=torch.zeros((2, 1, 64, 64), dtype=torch.bfloat16, device=DEV), page_size=64, ring=0, writes=True, has_values=True)
    whole = SimpleNamespace(longest=129, most_new=5)
    x = torch.zeros((5, 196), dtype=torch.bfloat16, device=DEV)
    assert ops.extends_in_pages(x[:, :192].contiguous(), 64, line, whole)
    assert not ops.extends_in_pages(x[:, :192], 64, line, whole) and not ops.extends_in_pages(torch.zeros(5 * 192 + 4, dtype=torch.bfloat16, device=DEV)[4:].view(5, 192), 64, line, whole)
