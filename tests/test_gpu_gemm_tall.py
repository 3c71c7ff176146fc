"""Products tall enough for any tile to fill the GPU, at the output widths where the
rule for the tile's width turns: against float64, errors of FP32 accumulation."""
import pytest
import torch

from espec_b200 import warmstart as WS

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("N", [1, 32, 33, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("M,K", [(18944, 40), (18945, 136)])
def test_tall(M, K, N):
    g = torch.Generator(device=DEV).manual_seed(N)
    A = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    B = torch.randn(K, N, generator=g, device=DEV).to(torch.bfloat16)
    exact = A.double() @ B.double()
    # K products, exact in FP32, summed with K roundings of 2^-24 of the partial sums
    bound = K * 2.0 ** -24 * (A.double().abs() @ B.double().abs())
    assert bool(((WS.gemm_bf16(A, B).double() - exact).abs() <= bound).all())
