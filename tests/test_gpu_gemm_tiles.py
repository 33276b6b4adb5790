"""Whole-prompt products with tiles of 256, 128 and 64 columns: an element's sum runs over the inner size in one order whatever the
tile, so every width gives the same bits, and so do the same rows among many."""
import pytest
import torch

from quicknn_b200.kernels import ops
from quicknn_b200.kernels.lib import KernelError, load

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MANY = 20000             # rows for more tiles than there are pairs of SMs, whatever their width


@pytest.mark.parametrize("M", [129, 256, 257, 640, 1025, 2048])
@pytest.mark.parametrize("N,K", [(8, 1024), (64, 64), (72, 2304), (256, 1160), (264, 136), (768, 2304), (2304, 2048), (2304, 9216), (4100, 520)])
def test_tile_widths(M, N, K):
    torch.manual_seed(M + N + K)
    x, w = torch.randn((MANY, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * 0.05).bfloat16()
    many = ops.gemm_tcgen05(x, w, tile_cols=256)
    act = ops.gemm_tcgen05(x, w, epilogue=ops.EPI_ACT, activation="silu", tile_cols=256)
    want = x[:M].double() @ w.double().T
    assert ((many[:M].double() - want).norm() / want.norm()).item() < 2e-3       # bfloat16's own rounding
    for cols in (0, 64, 128, 256):
        out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)      # nothing is written behind the last row
        got = ops.gemm_tcgen05(x[:M], w, out=out[:M], tile_cols=cols)
        assert (out[M] == 7.0).all() and torch.equal(got, many[:M]), cols
        assert torch.equal(ops.gemm_tcgen05(x[:M], w, epilogue=ops.EPI_ACT, activation="silu", tile_cols=cols), act[:M]), cols
    ops.raise_on_status(torch.device(DEV))


@pytest.mark.parametrize("cols,epilogue", [(32, ops.EPI_NONE), (192, ops.EPI_NONE), (-64, ops.EPI_NONE), (128, ops.EPI_GATED)])
def test_other_widths_are_refused(cols, epilogue):
    x = torch.zeros((256, 64), dtype=torch.bfloat16, device=DEV)
    with pytest.raises(KernelError):
        ops.gemm_tcgen05(x, x, epilogue=epilogue, tile_cols=cols)


@pytest.mark.parametrize("cols", range(64, 257, 32))
def test_chosen_widths(cols):
    """Every width that is chosen by itself, at products that it is chosen for: the bits of 256 columns."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chosen = load().qnn_gemm_tcgen05_2cta_cols
    sizes = [(M, N) for M in range(200, 3000, 200) for N in range(8, 4400, 8) if chosen(M, N, sms) == cols]
    K = 328
    for M, N in (sizes[0], sizes[len(sizes) // 2], sizes[-1]):
        torch.manual_seed(M + N)
        x, w = torch.randn((M - 3, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * 0.05).bfloat16()
        out = torch.full((M - 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
        got = ops.gemm_tcgen05(x, w, out=out[:M - 3])
        assert torch.equal(got, ops.gemm_tcgen05(x, w, tile_cols=256)) and (out[M - 3] == 7.0).all(), (M, N)
    ops.raise_on_status(torch.device(DEV))


@pytest.mark.parametrize("K", [72, 776, 2312])
@pytest.mark.parametrize("cols", range(64, 257, 32))
def test_chosen_widths_by_inner_size(cols, K):
    """The same with the inner size that the choice counts."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    width = load().qnn_gemm_tcgen05_2cta_width
    sizes = [(M, N) for M in range(200, 4400, 300) for N in range(8, 4400, 8) if width(M - 3, N, K, sms) == cols]
    assert sizes or K < 2312
    for M, N in {sizes[0], sizes[len(sizes) // 2], sizes[-1]} if sizes else ():
        torch.manual_seed(M + N)
        x, w = torch.randn((M - 3, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * 0.05).bfloat16()
        out = torch.full((M - 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
        got = ops.gemm_tcgen05(x, w, out=out[:M - 3])
        assert torch.equal(got, ops.gemm_tcgen05(x, w, tile_cols=256)) and (out[M - 3] == 7.0).all(), (M, N)
    ops.raise_on_status(torch.device(DEV))
