"""Whole-prompt products with tiles of 256, 128 and 64 columns: an element's sum runs over the inner size in one order whatever the
tile, so a product of few rows (narrow tiles) gives bit for bit what the same rows give among many (tiles of 256 columns)."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MANY = 20000             # rows from which every product here takes tiles of 256 columns


@pytest.mark.parametrize("M", [129, 256, 257, 640, 1025, 2048])
@pytest.mark.parametrize("N,K", [(8, 1024), (64, 64), (72, 2304), (256, 1160), (264, 136), (768, 2304), (2304, 2048), (2304, 9216), (4100, 520)])
def test_narrow_tiles(M, N, K):
    torch.manual_seed(M + N + K)
    x, w = torch.randn((MANY, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * 0.05).bfloat16()
    many = ops.gemm_tcgen05(x, w)
    out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)          # nothing is written behind the last row
    got = ops.gemm_tcgen05(x[:M], w, out=out[:M])
    assert (out[M] == 7.0).all() and torch.equal(got, many[:M])
    want = x[:M].double() @ w.double().T
    assert ((got.double() - want).norm() / want.norm()).item() < 2e-3            # bfloat16's own rounding
    assert torch.equal(ops.gemm_tcgen05(x[:M], w, epilogue=ops.EPI_ACT, activation="silu"),
                       ops.gemm_tcgen05(x, w, epilogue=ops.EPI_ACT, activation="silu")[:M])
    ops.raise_on_status(torch.device(DEV))
