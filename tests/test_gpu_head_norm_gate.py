"""The norm per head with a gate: head sizes around the steps of what a lane holds, heads that are no multiple of a warp's lanes, every kind
of weight, gate and denominator, float32 and bfloat16."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("vdim", [1, 31, 33, 100, 128, 129, 256, 257, 300, 511, 512, 600])
@pytest.mark.parametrize("T,H", [(1, 1), (5, 3), (130, 9)])
@pytest.mark.parametrize("act,weights,den", [("silu", "head", False), ("sigmoid", "row", True), ("none", None, False), ("silu", None, True), ("none", "row", True)])
@pytest.mark.parametrize("dt", ["bfloat16", "float32"])
def test_head_norm_gate(vdim, T, H, act, weights, den, dt):
    if weights == "head" and H == 1:
        weights = "row"
    torch.manual_seed(vdim + T + H)
    dt, hs, eps, g_col = getattr(torch, dt), vdim + 3, 1e-5, 8
    o = torch.randn((T, H, hs), device=DEV)
    o[:, :, vdim + 1:] = float("nan")                             # behind the normaliser: nothing to read
    w = None if weights is None else torch.randn(vdim if weights == "head" else H * vdim, device=DEV)
    e = torch.rand((T, 2 * H), device=DEV) if den else None
    gate = None if act == "none" else torch.randn((T, g_col + H * vdim + 5), device=DEV).to(dt)
    got = ops.head_norm_gate(o.view(T, H * hs), hs, H, vdim, eps, gate, 0 if gate is None else g_col, act, weight=w, den=e, den_col=H if den else 0,
                             out_dtype=dt if gate is None else None)
    y = o[:, :, :vdim].double()
    if den:
        y = y / (torch.maximum(o[:, :, vdim].abs(), e[:, H:]).double() + 1e-6)[:, :, None]
    y = y * torch.rsqrt((y * y).mean(-1, keepdim=True) + eps)
    if w is not None:
        y = y * w.double().view(-1, vdim)
    if gate is not None:
        z = gate[:, g_col:g_col + H * vdim].double().view(T, H, vdim)
        y = y * torch.sigmoid(z) * (z if act == "silu" else 1.0)
    y = y.reshape(T, -1)
    # float32 throughout: a sum of up to 600 squares, a root, an exponential; then the result's own rounding
    assert got.dtype == dt and ((got.double() - y).norm() / y.norm()).item() < (2.0 ** -8 if dt == torch.bfloat16 else 1e-6)
