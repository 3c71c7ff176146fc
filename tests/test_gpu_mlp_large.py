"""Conversions, column sums and losses on both sides of the line (4096 CTAs) from which
they run without overlapping their neighbours: exact conversions; sums in float64; and a
mixed chain, where a kernel of either kind follows the other."""
import pytest
import torch

from espec_b200 import _native as N
from espec_b200 import warmstart as WS

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("n", [1, 4096 * 256, 4096 * 256 + 1, 5_000_001])
def test_conversion(n):
    x = torch.randn(n, device=DEV)
    assert torch.equal(WS.to_bf16(x), x.to(torch.bfloat16))


@pytest.mark.parametrize("rows,cols", [(9, 4096 * 32), (9, 4096 * 32 + 1), (4096, 33), (4097, 33)])
def test_sums(rows, cols):
    lib, st = N.load(), torch.cuda.current_stream().cuda_stream
    y, t = torch.randn(rows, cols, device=DEV), torch.randn(rows, cols, device=DEV)
    db, dy = torch.empty(cols, device=DEV), torch.empty(rows, cols, device=DEV)
    loss = torch.empty(rows, device=DEV)
    N.check(lib.espec_mlp_colsum(y.data_ptr(), rows, cols, db.data_ptr(), st), "colsum")
    N.check(lib.espec_mlp_mse(y.data_ptr(), t.data_ptr(), rows, cols, dy.data_ptr(),
                              loss.data_ptr(), st), "mse")
    # at most `rows` (`cols`) FP32 roundings of sums of magnitudes
    assert bool(((db - y.double().sum(0)).abs() <= rows * 2.0 ** -24 * y.double().abs().sum(0)).all())
    d = y.double() - t.double()
    want = (d * d).sum(1) / d.numel()
    assert bool(((loss - want).abs() <= (cols + 4) * 2.0 ** -23 * want).all())
    assert bool(((dy - 2 * d / d.numel()).abs() <= 4 * 2.0 ** -24 * (2 * d / d.numel()).abs() +
                 2.0 ** -23 * (y.abs() + t.abs()).double() / d.numel()).all())


def test_mixed_chain():
    small, large = 512, 4096 * 256 + 512
    x = torch.zeros(large, device=DEV)
    a = torch.empty(small, dtype=torch.bfloat16, device=DEV)
    b = torch.empty(large, dtype=torch.bfloat16, device=DEV)
    for k in range(1, 200):
        x.fill_(float(k))
        WS.to_bf16(x[:small], a)
        WS.to_bf16(x, b)
        WS.to_bf16(x[large - small:], a)
    assert bool((a == torch.tensor(199.0, dtype=torch.bfloat16)).all())
    assert bool((b == torch.tensor(199.0, dtype=torch.bfloat16)).all())
