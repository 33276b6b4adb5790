"""Bias, head norms and rotation of packed rows: heads of every number of lanes, with and without a norm of queries or keys, weights
that start off 16 bytes, norms over part of a head, more heads than a block's warps hold."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def exact(x, nq, nk, hd, bias, wq, wk, norm_dim, eps, rot, freq, pos, interleaved):
    T = x.shape[0]
    y = x.double() if bias is None else x.double() + bias.double()
    heads = y[:, :(nq + nk) * hd].reshape(T, nq + nk, hd).clone()
    for lo, hi, w in ((0, nq, wq), (nq, nq + nk, wk)):
        if w is not None and hi > lo:
            h = heads[:, lo:hi, :norm_dim]
            heads[:, lo:hi, :norm_dim] = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + eps) * w.double()
    if rot:
        a = (pos.float()[:, None] * freq[None, :]).double()[:, None, :]
        one, two = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
        u, v = heads[..., one].clone(), heads[..., two].clone()
        heads[..., one], heads[..., two] = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
    return torch.cat([heads.reshape(T, -1), y[:, (nq + nk) * hd:]], 1)


@pytest.mark.parametrize("T", [1, 33, 1025])
@pytest.mark.parametrize("nq,nk,hd", [(1, 1, 8), (3, 1, 64), (5, 5, 72), (12, 12, 64), (8, 4, 128), (7, 0, 136), (2, 2, 256)])
@pytest.mark.parametrize("norms,part,off", [("qk", False, 0), ("q", False, 0), ("k", True, 0), ("qk", True, 1), ("", False, 0)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_head_prep(T, nq, nk, hd, norms, part, off, interleaved):
    torch.manual_seed(T + nq + hd)
    norm_dim = hd - 3 if part else hd
    rot = hd // 16 * 16 if not interleaved else hd - 2
    x = torch.randn((T, (nq + 2 * nk) * hd), device=DEV).bfloat16()
    bias = torch.randn(x.shape[1], device=DEV)
    weight = lambda: torch.randn(norm_dim + off, device=DEV).bfloat16()[off:]  # noqa: E731
    wq, wk = (weight() if "q" in norms else None), (weight() if "k" in norms and nk else None)
    freq, pos = torch.rand(rot // 2, device=DEV), torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    dst = torch.empty(x.shape, dtype=torch.float32, device=DEV)
    got = ops.head_prep(x, 0, nq, nk, nk * hd, hd, dst=dst, bias=bias, q_norm=wq, k_norm=wk, norm_dim=norm_dim if wq is not None or wk is not None else 0,
                        eps=1e-6, rot_dim=rot, inv_freq=freq if rot else None, interleaved=interleaved, tok_pos=pos if rot else None)
    want = exact(x, nq, nk, hd, bias, wq, wk, norm_dim, 1e-6, rot, freq, pos, interleaved)
    # float32 throughout: sums of up to 256 squares, a root, a sine and a cosine
    assert ((got.double() - want).norm() / want.norm()).item() < 1e-6
