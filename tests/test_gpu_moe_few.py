"""Experts of a few rows each (tiles of up to 16 rows): one row to a whole tile and one more, inner sizes of one block of 32 to more
than are kept in flight, columns that are no whole number of a block's, the score on the input and on the output.  Oracle: the
same in 64 bits with the hidden rows rounded to bfloat16 where the kernels round them (2^-8 relative, summed over the inner size)."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,E,top", [(1, 4, 1), (3, 5, 2), (8, 16, 2), (17, 2, 1), (33, 2, 2)])
@pytest.mark.parametrize("W,ff", [(32, 32), (96, 64), (160, 288), (2304, 576)])
@pytest.mark.parametrize("on_input,gated", [(True, True), (False, True), (False, False)])
def test_few_rows(T, E, top, W, ff, on_input, gated):
    torch.manual_seed(T + W)
    nm = 2 if gated else 1
    x = torch.randn((T, W), device=DEV).bfloat16()
    wgu, wd = (torch.randn(s, device=DEV).mul_(W ** -0.5).bfloat16() for s in ((E, nm * ff, W), (E, W, ff)))
    sel_e = torch.stack([torch.randperm(E, device=DEV)[:top] for _ in range(T)]).int().contiguous()
    sel_w = torch.rand((T, top), device=DEV) + 0.25
    got = ops.moe_experts(x, sel_e, sel_w, top, wgu, wd, ops.ACT_CODES["silu"], 0.0, 1.0, on_input, grouped=False, gated=gated)
    want = torch.zeros((T, W), dtype=torch.float64, device=DEV)
    for t in range(T):
        for k in range(top):
            e, s = int(sel_e[t, k]), sel_w[t, k]
            row = (x[t].float() * s).bfloat16().double() if on_input else x[t].double()
            up = wgu[e].double() @ row
            h = torch.nn.functional.silu(up[:ff]) * (up[ff:] if gated else 1.0)
            y = wd[e].double() @ h.bfloat16().double()
            want[t] += y if on_input else y * s.double()
    assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8
