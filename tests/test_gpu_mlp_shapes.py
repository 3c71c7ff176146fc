"""The network's calls refuse tensors of another width, batch, element size or memory
than theirs before anything is launched, and take what is left after a refusal."""
import pytest
import torch

from espec_b200 import warmstart as WS

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
SIZES = [5, 64, 48, 96]


@pytest.fixture(scope="module")
def net():
    return WS.MLP(SIZES, seed=3, device=DEV)


def ones(rows, cols, dtype, dev=DEV):
    return torch.ones((rows, cols), dtype=dtype, device=dev)


BF, F = torch.bfloat16, torch.float32


@pytest.mark.parametrize("x", [(32, 4, BF), (32, 6, BF), (32, 5, F), (32, 5, torch.uint8)], ids=str)
def test_forward_refuses(net, x):
    with pytest.raises(AssertionError):
        net.forward(ones(*x))
    with pytest.raises(AssertionError):
        net.forward(torch.ones(5, dtype=BF, device=DEV))


@pytest.mark.parametrize("which", ["dy_rows", "dy_cols", "dy_type", "h_rows", "h_cols", 
                                   "h_type", "h_host", "z_rows", "z_cols", "z_short",
                                   "h_short"])
def test_backward_refuses(net, which):
    hs, zs = net.forward(ones(32, 5, BF))
    dY = ones(32, SIZES[-1], F)
    if which == "dy_rows":
        dY = ones(33, SIZES[-1], F)
    elif which == "dy_cols":
        dY = ones(32, SIZES[-1] + 1, F)
    elif which == "dy_type":
        dY = ones(32, SIZES[-1], BF)
    elif which[0] == "h":
        hs = {"rows": [hs[0], ones(31, 64, BF), hs[2]], "cols": [hs[0], ones(32, 63, BF), hs[2]],
              "type": [hs[0], ones(32, 64, torch.uint8), hs[2]],
              "host": [hs[0].cpu(), *hs[1:]], "short": hs[:2]}[which[2:]]
    else:
        zs = {"rows": [zs[0], ones(16, 48, F), zs[2]], "cols": [zs[0], ones(32, 40, F), zs[2]],
              "short": zs[:1]}[which[2:]]
    with pytest.raises(AssertionError):
        net.backward(hs, zs, dY)


def test_accepted(net):
    wide = torch.randn(32, 10, device=DEV).to(BF)
    x = wide[:, ::2]  # strided input: taken as its values
    hs, zs = net.forward(x)
    hs2, zs2 = net.forward(x.contiguous())
    assert all(torch.equal(a, b) for a, b in zip(hs + zs, hs2 + zs2))
    dY = torch.randn(32, SIZES[-1], device=DEV)
    g = net.backward(hs, zs, dY)
    g2 = net.backward(hs, zs[:-1], dY)  # the output itself is not read
    assert all(torch.equal(a, b) for a, b in zip(g, g2)) and len(g) == 6
    g2 = net.backward(hs, zs, dY.t().contiguous().t())  # a strided gradient: its values
    assert all(torch.equal(a, b) for a, b in zip(g, g2))
