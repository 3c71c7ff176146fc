"""The eigensolver's forms -- two CTAs per potential, one, the vector in shared or
global memory -- add in the same order: one potential alone (two CTAs from 2048 points
on) and the same one among 80 (one CTA each) give the same bits; H v = E v to the
solver's tolerance."""
import pytest
import torch

from espec_b200 import eig as EG

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("np_", [(45, 45), (32, 64), (43, 48), (61, 67), (160, 154)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_alone_and_in_a_batch(np_):
    g = EG.Grid2D(np_)
    nb = 80 if g.n < 20000 else 3
    q = torch.tensor([0.17, 1.0, 0.12, 1.2, 0.01], dtype=torch.float64, device=DEV).repeat(nb, 1)
    q[1:, 0] += 0.0005 * torch.arange(1, nb, device=DEV)
    v = EG.morse2d_potentials(g, q)
    st = EG.lcg_start(g.n, 2, DEV).expand(nb, 2, g.n).contiguous()
    kw = dict(nstates=2, m=24, tol=1e-8, maxrest=400)
    many = EG.solve(g, v, st, **kw)
    one = EG.solve(g, v[:1].contiguous(), st[:1].contiguous(), **kw)
    assert bool((many["resid"] <= 1e-8).all())
    for key in ("eval", "vec", "resid", "matvecs"):
        assert torch.equal(many[key][:1], one[key]), key
