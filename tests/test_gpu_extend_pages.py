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
