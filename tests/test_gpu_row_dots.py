"""Gates per head, router logits and products with few outputs of a prompt's many rows (8 or 64 rows a block) beside those of few rows:
as far from 64 bits as float32 sums are, whatever the width, the outputs and the rows left over, and the same bits however many rows a
step has."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MANY = 256


def off(a, want):
    return ((a.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("T", [MANY, MANY + 1, MANY + 7, 700])
@pytest.mark.parametrize("W,E,extra", [(8, 2, 0), (40, 16, 1), (264, 17, 0), (1536, 31, 1), (2304, 16, 0), (2304, 32, 0)])
@pytest.mark.parametrize("score", ["sigmoid", "softmax"])
def test_route(T, W, E, extra, score):
    torch.manual_seed(T + W + E)
    x, w = torch.randn((T, W), device=DEV).bfloat16(), (torch.randn((E + extra, W), device=DEV) * 2 * W ** -0.5).bfloat16()
    z = x.double() @ w.double().T
    s = torch.sigmoid(z[:, :E]) if score == "sigmoid" else z[:, :E].softmax(-1)
    top = min(2, E)
    res = ops.moe_route(x, w, top, score, False, **({"extra": extra} if extra else {}))
    sel_e, sel_w = res[0].view(T, top).long(), res[1].view(T, top)
    assert (sel_e >= 0).all() and (sel_e < E).all() and (sel_e.sort(-1).values.diff(dim=-1) > 0).all()
    want = s.gather(1, sel_e)
    best = s.topk(top, -1).values
    assert off(sel_w, want) < 1e-6 and ((best - want).abs() <= 1e-6 * best.abs() + 1e-7).all()         # the best, ties by rounding aside
    if extra:
        assert off(res[2], z[:, E:]) < 1e-6
    few = [ops.moe_route(x[lo:lo + 100].contiguous(), w, top, score, False, **({"extra": extra} if extra else {})) for lo in range(0, T, 100)]
    same = torch.cat([f[0] for f in few]).view(T, top).long() == sel_e
    assert same.float().mean().item() > 0.999


@pytest.mark.parametrize("T", [1024, 1025, 1500])
@pytest.mark.parametrize("W,H,D", [(8, 1, 8), (264, 9, 256), (1536, 12, 64), (2304, 16, 8), (2304, 17, 128), (2304, 32, 16)])
@pytest.mark.parametrize("dt", ["bfloat16", "float32"])
def test_gate_heads(T, W, H, D, dt):
    torch.manual_seed(T + W + H)
    x, w = torch.randn((T, W), device=DEV).bfloat16(), (torch.randn((H, W), device=DEV) * W ** -0.5).bfloat16()
    o = torch.randn((T, H * D), device=DEV).to(getattr(torch, dt))
    want = (o.double().view(T, H, D) * torch.sigmoid(x.double() @ w.double().T)[:, :, None]).view(T, -1)
    few = torch.cat([ops.gate_heads(o[lo:lo + 100].clone(), x[lo:lo + 100].contiguous(), w, H) for lo in range(0, T, 100)])
    got = ops.gate_heads(o.clone(), x, w, H)
    if dt == "float32":
        assert off(got, want) < 2e-7 and off(got, want) < 1.1 * off(few, want) + 1e-8
    else:
        assert off(got, want) < 2.0 ** -8


def test_values_that_are_not_finite_stay_in_their_row():
    T, W, H, D = 1030, 264, 9, 16
    torch.manual_seed(1)
    x, w = torch.randn((T, W), device=DEV).bfloat16(), torch.randn((H, W), device=DEV).bfloat16()
    o = torch.randn((T, H * D), device=DEV)
    clean = ops.gate_heads(o.clone(), x, w, H)
    x[17, 3], x[42, 100] = float("nan"), float("inf")
    got = ops.gate_heads(o.clone(), x, w, H)
    others = torch.tensor([t not in (17, 42) for t in range(T)], device=DEV)
    assert torch.equal(got[others], clean[others]) and got[17].isnan().all()


@pytest.mark.parametrize("T", [MANY, MANY + 1, 700])
@pytest.mark.parametrize("K,N", [(136, 1), (1536, 24), (2304, 32), (264, 17), (8, 700), (64, 1152), (72, 577), (128, 640)])
@pytest.mark.parametrize("decay", [False, True])
def test_small_linear(T, K, N, decay):
    """Long rows with few outputs, short rows with many."""
    torch.manual_seed(T + K + N)
    x, w = torch.randn((T, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * K ** -0.5).bfloat16()
    bias = torch.randn(N, device=DEV)
    kw = dict(decay_bias=bias, tau=8.0) if decay else {}
    z = x.double() @ w.double().T
    want = torch.sigmoid(z + bias.double()) ** 0.125 if decay else z
    got = ops.small_linear_f32(x, w, **kw)
    few = torch.cat([ops.small_linear_f32(x[lo:lo + 100].contiguous(), w, **kw) for lo in range(0, T, 100)])
    assert off(got, want) < 2e-7 and off(got, want) < 1.1 * off(few, want) + 1e-8


def pieces(T):
    """A step's rows as other steps might bring them: one alone, a few, the rest in hundreds."""
    cuts = [0, 1, 2, 9] + list(range(100, T, 100)) + [T]
    return list(zip(cuts[:-1], cuts[1:]))


@pytest.mark.parametrize("T", [255, MANY, MANY + 1, MANY + 7, 2050])
@pytest.mark.parametrize("W,E,extra", [(8, 4, 0), (264, 20, 1), (1536, 32, 0), (2304, 16, 0), (2304, 31, 1), (1536, 36, 0)])
def test_route_does_not_depend_on_the_rows_beside(T, W, E, extra):
    torch.manual_seed(T + W + E)
    x, w = torch.randn((T, W), device=DEV).bfloat16(), (torch.randn((E + extra, W), device=DEV) * 2 * W ** -0.5).bfloat16()
    kinds = [dict(score="sigmoid"), dict(score="softmax", renormalize=True)]
    if E % 4 == 0 and E > 4:
        kinds.append(dict(score="sigmoid", renormalize=True, correction=torch.randn(E, device=DEV), scale=2.5, groups=(4, 2)))
    for kw in kinds:
        kw.update({"extra": extra} if extra else {})
        whole = ops.moe_route(x, w, 2, **kw)
        parts = [ops.moe_route(x[lo:hi].contiguous(), w, 2, **kw) for lo, hi in pieces(T)]
        for i, res in enumerate(whole):
            assert torch.equal(torch.cat([p[i] for p in parts]), res), (kw, i)


@pytest.mark.parametrize("T", [1023, 1024, 1025, 2050])
@pytest.mark.parametrize("W,H,D", [(8, 1, 8), (264, 9, 256), (1536, 31, 8), (2304, 32, 16), (2304, 33, 16)])
def test_gates_do_not_depend_on_the_rows_beside(T, W, H, D):
    torch.manual_seed(T + W + H)
    x, w = torch.randn((T, W), device=DEV).bfloat16(), (torch.randn((H, W), device=DEV) * W ** -0.5).bfloat16()
    o = torch.randn((T, H * D), device=DEV).bfloat16()
    parts = [ops.gate_heads(o[lo:hi].clone(), x[lo:hi].contiguous(), w, H, 0.7) for lo, hi in pieces(T)]
    assert torch.equal(torch.cat(parts), ops.gate_heads(o.clone(), x, w, H, 0.7))


@pytest.mark.parametrize("K,N,Ts", [(136, 1, (511, 512, 513, 519)), (1536, 24, (511, 512, 513, 519)), (2304, 32, (512, 2050)), (1536, 33, (513,)),
                                    (8, 700, (63, 64, 65, 255, 700)), (64, 1152, (127, 137, 256, 700)), (33, 577, (257, 700)), (128, 640, (256, 1500)),
                                    (100, 65, (2050,))])
@pytest.mark.parametrize("dtypes", [("bfloat16", "bfloat16"), ("bfloat16", "float32"), ("float32", "float32")])
@pytest.mark.parametrize("decay", [False, True])
def test_small_linear_does_not_depend_on_the_rows_beside(K, N, Ts, dtypes, decay):
    for T in Ts:
        torch.manual_seed(T + K + N)
        x, w = torch.randn((T, K), device=DEV).to(getattr(torch, dtypes[0])), (torch.randn((N, K), device=DEV) * K ** -0.5).to(getattr(torch, dtypes[1]))
        kw = dict(decay_bias=torch.randn(N, device=DEV), tau=8.0) if decay else {}
        parts = [ops.small_linear_f32(x[lo:hi].contiguous(), w, **kw) for lo, hi in pieces(T)]
        assert torch.equal(torch.cat(parts), ops.small_linear_f32(x, w, **kw)), T
