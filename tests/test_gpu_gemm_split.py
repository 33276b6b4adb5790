"""Whole-prompt products whose tiles are shared by several pairs of CTAs: one tile to as many as the device holds at once and one
more, inner sizes whose slabs do not part evenly, ragged rows and columns, an activation.  Oracle: the product in 64 bits; a
bfloat16 result is off by its own rounding (2^-9 relative, 1.7e-3 in the 2-norm) and float32 sums (1e-6)."""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M", [129, 256, 257, 640, 1025])
@pytest.mark.parametrize("N,K", [(8, 1024), (64, 2304), (256, 1160), (264, 8 * 129), (768, 2304), (2304, 2048), (2304, 9216), (4096, 4104)])
def test_shared_tiles(M, N, K):
    torch.manual_seed(M + N + K)
    x, w = torch.randn((M, K), device=DEV).bfloat16(), (torch.randn((N, K), device=DEV) * 0.05).bfloat16()
    want = x.double() @ w.double().T
    out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)          # nothing is written behind the last row
    got = ops.gemm_tcgen05(x, w, out=out[:M])
    assert got is not None and (out[M] == 7.0).all()
    assert ((got.double() - want).norm() / want.norm()).item() < 2e-3
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()
    assert (ops.gemm_tcgen05(x, w) == got).all()                                 # whichever pair comes last
    act = ops.gemm_tcgen05(x, w, epilogue=ops.EPI_ACT, activation="relu2")
    relu2 = want.clamp(min=0) ** 2
    assert ((act.double() - relu2).norm() / relu2.norm()).item() < 4e-3          # the square doubles a relative error
    ops.raise_on_status(torch.device(DEV))
