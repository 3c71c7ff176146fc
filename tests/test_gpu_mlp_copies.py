"""A network can be saved, pickled and deep-copied; the copy computes the same bits."""
import copy
import io
import pickle

import pytest
import torch

from espec_b200 import warmstart as WS

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def saved(net):
    f = io.BytesIO()
    torch.save(net, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


@pytest.mark.parametrize("how", ["save", "pickle", "deepcopy"])
def test_copy(how):
    net = WS.MLP([5, 32, 48, 64], seed=1, device=DEV)
    other = {"save": saved, "pickle": lambda n: pickle.loads(pickle.dumps(n)),
             "deepcopy": copy.deepcopy}[how](net)
    x = torch.randn(32, 5, device=DEV).to(torch.bfloat16)
    t = torch.randn(32, 64, device=DEV)
    out = []
    for n in (net, other):
        hs, zs = n.forward(x)
        out.append([*zs, *n.backward(hs, zs, n.loss_grad(zs[-1], t)[1])])
    assert all(torch.equal(a, b) for a, b in zip(*out))
