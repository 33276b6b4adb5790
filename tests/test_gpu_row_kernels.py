"""Row kernels that take eight elements per thread, and those that walk a row, at the sizes where the way changes: the smallest
rows, rows that are no whole number of warps, the largest, eight elements more, and rows that do not start on 16 bytes.

Tolerance: sums of up to 8192 float32 terms by a tree (about 2^-24 sqrt(13)) and a few roundings: 2e-6 of the row's largest value;
bfloat16 results one rounding of 2^-8."""
import pytest
import torch

from quicknn_b200.kernels import ops
from quicknn_b200.kernels.lib import NonFiniteLogits

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WIDTHS = [8, 24, 256, 264, 2304, 4096, 4104, 8184, 8192, 8200, 100, 2305]


def close(got, want, dtype=torch.float32):
    tol = 2e-6 if dtype == torch.float32 else 2 ** -8
    assert ((got.double() - want).abs().amax(-1) <= tol * want.abs().amax(-1).clamp(min=1e-30)).all()


def rms(x, eps):
    return x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt()


def layernorm(x, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / (d.pow(2).mean(-1, keepdim=True) + eps).sqrt()


@pytest.mark.parametrize("W", WIDTHS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 9])
def test_norms_and_adds(W, dtype, T):
    torch.manual_seed(W + T)
    mk = lambda *s: torch.randn(s, device=DEV).to(dtype)  # noqa: E731
    x, y, z, w, b = mk(T, W), mk(T, W), mk(T, W), mk(W), mk(W)
    stream = torch.randn((T, W), device=DEV)
    D = lambda t: t.double()  # noqa: E731
    close(ops.rmsnorm(x, w, 1e-6, True, dtype), rms(D(x), 1e-6) * (1 + D(w)), dtype)
    r = stream.clone()
    want = D(stream) + 0.5 * D(y)
    out = ops.add_scaled_rmsnorm(r, y, 0.5, w, 1e-6, False, dtype)
    close(r, want)
    close(out, rms(want, 1e-6) * D(w), dtype)
    close(ops.layernorm(x, w, 1e-5, dtype), layernorm(D(x), 1e-5) * D(w), dtype)
    r = stream.clone()
    copy = ops.add_layernorm(r, y, w, 1e-5, bias=b, copy_dtype=dtype)
    want = D(stream) + layernorm(D(y) + D(b), 1e-5) * D(w)
    close(r, want)
    close(copy, want, dtype)
    r = stream.clone()
    copy = ops.add_mean_layernorm(r, [y, z], [b, w], 1e-6, w, 1e-5, dtype)
    want = D(stream) + layernorm((rms(D(y), 1e-6) * D(b) + rms(D(z), 1e-6) * D(w)) / 2, 1e-5) * D(w)
    close(r, want)
    close(copy, want, dtype)
    table = mk(7, W)
    ids = torch.arange(T, dtype=torch.int32, device=DEV) % 7
    close(ops.embed(ids, table, 3.0), 3.0 * D(table)[ids.long()])


@pytest.mark.parametrize("T", [383, 384, 385])
@pytest.mark.parametrize("W", [8, 2304, 2305])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_of_many_rows(T, W, dtype):
    torch.manual_seed(T)
    table = torch.randn((50, W), device=DEV).to(dtype)
    ids = torch.randint(0, 50, (T,), dtype=torch.int32, device=DEV)
    assert torch.equal(ops.embed(ids, table, 3.0), 3.0 * table.float()[ids.long()])


# (columns of the rows, first column, of the result's rows, first columns): eights on 16 bytes; then a pitch or a first column that is not
PIECES = [(2048, 256, 1024, 64, 576), (264, 8, 520, 0, 264), (1032, 8, 1032, 8, 520), (2049, 8, 1024, 64, 576), (2048, 3, 1024, 64, 576),
          (2048, 256, 1028, 64, 576), (2048, 256, 1024, 60, 576), (2048, 256, 1024, 64, 577), (1028, 4, 1028, 4, 516)]


@pytest.mark.parametrize("ldx,col,ldo,out1,out2", PIECES)
@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("T", [1, 9])
@pytest.mark.parametrize("twice", [False, True])
def test_pieces_of_rows(ldx, col, ldo, out1, out2, dtype, out_dtype, T, twice):
    n = 256
    torch.manual_seed(ldx + col)
    x, w = torch.randn((T, ldx), device=DEV).to(dtype), torch.randn(n, device=DEV).to(dtype)
    out = torch.full((T, ldo), 7.0, device=DEV).to(out_dtype)
    ops.rmsnorm_cols(x, col, n, w, 1e-6, out, out1, out2 if twice else None)
    want = rms(x[:, col:col + n].double(), 1e-6) * w.double()
    rest = torch.ones(ldo, dtype=torch.bool, device=DEV)
    for at in [out1] + ([out2] if twice else []):
        close(out[:, at:at + n], want, out_dtype)
        rest[at:at + n] = False
    assert (out[:, rest] == 7.0).all()                               # and nothing beside the pieces
    if dtype == out_dtype:
        got = torch.full((T, ldo), 7.0, device=DEV).to(dtype)
        ops.copy_col_range(x, col, n, got, out1)
        keep = torch.full((T, ldo), 7.0, device=DEV).to(dtype)
        keep[:, out1:out1 + n] = x[:, col:col + n]
        assert torch.equal(got, keep)
        piece = x[:, col:col + n].contiguous()
        got.fill_(7.0)
        ops.copy_cols(piece, got, out1)
        assert torch.equal(got, keep)


@pytest.mark.parametrize("W", [8, 264, 4096, 4104, 100])
@pytest.mark.parametrize("branches", [1, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_and_four_branches(W, branches, dtype):
    torch.manual_seed(W)
    ys, ws = [torch.randn((5, W), device=DEV).to(dtype) for _ in range(branches)], [torch.randn(W, device=DEV).to(dtype) for _ in range(branches)]
    w, stream = torch.randn(W, device=DEV).to(dtype), torch.randn((5, W), device=DEV)
    r = stream.clone()
    ops.add_mean_layernorm(r, ys, ws, 1e-6, w, 1e-5)
    mean = sum(rms(y.double(), 1e-6) * v.double() for y, v in zip(ys, ws)) / branches
    close(r, stream.double() + layernorm(mean, 1e-5) * w.double())


@pytest.mark.parametrize("offset", [0, 1, 8])
@pytest.mark.parametrize("W", [8, 2304])
def test_rows_that_do_not_start_on_16_bytes(W, offset):
    """Widths of eights: only where the memory starts decides the way."""
    torch.manual_seed(W)
    take = lambda t: torch.cat([t.new_zeros(offset), t.reshape(-1)])[offset:].view(t.shape)  # noqa: E731
    for dtype in (torch.float32, torch.bfloat16):
        x, w = take(torch.randn((3, W), device=DEV).to(dtype)), take(torch.randn(W, device=DEV).to(dtype))
        r0 = take(torch.randn((3, W), device=DEV))
        close(ops.layernorm(x, w, 1e-5, dtype), layernorm(x.double(), 1e-5) * w.double(), dtype)
        r = take(r0)
        ops.add_layernorm(r, x, w, 1e-5)
        close(r, r0.double() + layernorm(x.double(), 1e-5) * w.double())
        r = take(r0)
        want = r0.double() + 0.5 * x.double()
        close(ops.add_scaled_rmsnorm(r, x, 0.5, w, 1e-6, False, torch.float32), rms(want, 1e-6) * w.double())
        close(r, want)


@pytest.mark.parametrize("inner", [8, 264, 2304, 33])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_clamped_gate(inner, dtype, offset):
    torch.manual_seed(inner)
    gu = (4 * torch.randn(7 * 2 * inner + offset, device=DEV)).to(dtype)[offset:].view(7, 2 * inner)
    g, u = gu.double().split(inner, 1)
    g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
    want = g * torch.sigmoid(1.7 * g) * (u + 1)
    close(ops.gated_act_clamped(gu, 7.0, 1.7), want, dtype)


def test_weights_that_the_kernel_in_front_writes():
    """A norm may follow the kernel that writes its weights, and reads what that kernel wrote."""
    torch.manual_seed(1)
    W, n, f32 = 2304, 4 << 20, torch.float32
    x, y, r0 = (torch.randn((4, W), device=DEV) for _ in range(3))
    out = torch.empty((4, W), device=DEV)
    for i in range(40):
        src = torch.randn(n, device=DEV).bfloat16()
        want = src[-2 * W:].float()
        torch.cuda.synchronize()
        w = ops.cast(src, f32)[-2 * W:-W]                        # its last blocks write what the norm reads
        got = [ops.layernorm(x, w, 1e-5, f32)]
        w, b = ops.cast(src, f32)[-2 * W:].split(W)
        got.append(r0.clone())                                   # (queued before the cast below)
        w, b = ops.cast(src, f32)[-2 * W:].split(W)
        ops.add_layernorm(got[1], y, w, 1e-5, bias=b)
        got.append(r0.clone())
        w = ops.cast(src, f32)[-W:]
        ops.add_mean_layernorm(got[2], [x, y], [x[0], y[0]], 1e-6, w, 1e-5)
        r = r0.clone()
        w = ops.cast(src, f32)[-W:]
        got.append(ops.add_scaled_rmsnorm(r, y, 0.5, w, 1e-6, False, f32))
        w = ops.cast(src, f32)[-W:]
        got.append(ops.rmsnorm_cols(x, 0, W, w, 1e-6, out).clone())
        D, v, b = (lambda t: t.double()), want[:W].double(), want[W:].double()
        close(got[0], layernorm(D(x), 1e-5) * v)
        close(got[1], D(r0) + layernorm(D(y) + b, 1e-5) * v)
        mean = (rms(D(x), 1e-6) * D(x[0]) + rms(D(y), 1e-6) * D(y[0])) / 2
        close(got[2], D(r0) + layernorm(mean, 1e-5) * b)
        close(got[3], rms(D(r0) + 0.5 * D(y), 1e-6) * b)
        close(got[4], rms(D(x), 1e-6) * b)


@pytest.mark.parametrize("n", [1, 3, 4, 4095, 4096, 4097, 1 << 20])
@pytest.mark.parametrize("bad", [None, float("nan"), float("inf"), float("-inf")])
def test_finite_check_sees_every_place(n, bad):
    for place in {0, n // 2, n - 1}:
        x = torch.zeros((1, n), device=DEV)
        if bad is not None:
            x[0, place] = bad
        ops.check_finite(x)
        if bad is None:
            ops.raise_on_status(torch.device(DEV))
        else:
            with pytest.raises(NonFiniteLogits):
                ops.raise_on_status(torch.device(DEV))


@pytest.mark.parametrize("K,N,T", [(64, 40, 128), (61, 33, 127), (128, 32, 200), (3, 1, 129), (136, 5, 3), (130, 5, 3),
                                   (64, 256, 592), (64, 256, 593), (61, 257, 640), (3, 1152, 140), (128, 1152, 129)])    # to 592 blocks of 8 rows, and beyond
def test_few_outputs(K, N, T):
    torch.manual_seed(K)
    x, w = torch.randn((T, K), device=DEV).bfloat16(), torch.randn((N, K), device=DEV).bfloat16()
    close(ops.small_linear_f32(x, w), x.double() @ w.double().T)
