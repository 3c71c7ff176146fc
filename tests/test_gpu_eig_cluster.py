"""Two CTAs of a cluster share one potential (2 x potentials <= SMs, 2048 points or
more): the sums of one restart and of the next follow each other with nothing but the
sums' own barriers between them.  Many short restarts of the first state, repeated, give
the bits of the one-CTA form every time."""
import pytest
import torch

from espec_b200 import eig as EG

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("nstates,m", [(1, 2), (1, 8), (3, 6)])
@pytest.mark.parametrize("np_", [(32, 64), (67, 61)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_restarts_repeat(np_, nstates, m):
    nsm = torch.cuda.get_device_properties(DEV).multi_processor_count
    few, many = nsm // 2, nsm
    g = EG.Grid2D(np_)
    q = torch.tensor([0.17, 1.0, 0.12, 1.2, 0.01], dtype=torch.float64, device=DEV).repeat(many, 1)
    q[:, 0] += 0.0002 * torch.arange(many, device=DEV)
    v = EG.morse2d_potentials(g, q)
    st = EG.lcg_start(g.n, nstates, DEV).expand(many, nstates, g.n).contiguous()
    kw = dict(nstates=nstates, m=m, tol=1e-3, maxrest=120)
    one = EG.solve(g, v, st, **kw)
    for _ in range(10):
        two = EG.solve(g, v[:few].contiguous(), st[:few].contiguous(), **kw)
        for key in ("eval", "vec", "resid", "matvecs"):
            assert torch.equal(one[key][:few], two[key]), key
