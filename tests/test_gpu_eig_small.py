"""The eigensolver on small grids, where a warp takes a whole product, up to the line for
the other form: eigenvalues of the dense matrix, and vectors with H v = E v."""
import numpy as np
import pytest
import torch

from espec_b200 import eig as EG

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def dense(g, v):
    """the 4th-order finite-difference H, x fastest"""
    def axis(n, s):
        a = np.zeros((n, n))
        for d, f in ((0, 30.0), (1, -16.0), (2, 1.0)):
            a += f * s * (np.eye(n, k=d) + (np.eye(n, k=-d) if d else 0.0))
        return a
    nx, ny = g.np
    return (np.kron(np.eye(ny), axis(nx, g.shm[0])) + np.kron(axis(ny, g.shm[1]), np.eye(nx))
            + np.diag(v))


@pytest.mark.parametrize("nprob", [1, 200])
@pytest.mark.parametrize("np_", [(5, 7), (8, 8), (16, 16), (31, 33), (32, 32), (33, 62), (32, 64)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_small(np_, nprob):
    g = EG.Grid2D(np_)
    q = torch.tensor([0.17, 1.0, 0.12, 1.2, 0.01], dtype=torch.float64, device=DEV)
    q = q.repeat(nprob, 1)
    q[:, 0] += 0.0001 * torch.arange(nprob, device=DEV)
    v = EG.morse2d_potentials(g, q)
    st = EG.lcg_start(g.n, 2, DEV).expand(nprob, 2, g.n).contiguous()
    r = EG.solve(g, v, st, nstates=2, m=min(30, g.n - 5), tol=1e-9, maxrest=400)
    assert bool((r["resid"] <= 1e-9).all())
    for p in (0, nprob - 1):
        H = dense(g, v[p].cpu().numpy())
        want = np.linalg.eigvalsh(H)[:2]
        # |E - E_exact| <= |H v - E v| for a symmetric H
        assert np.max(np.abs(r["eval"][p].cpu().numpy() - want)) <= 2e-9
        x = r["vec"][p].cpu().numpy()
        assert np.max(np.linalg.norm(x @ H - want[:, None] * x, axis=1)) <= 4e-9
        assert np.max(np.abs(x @ x.T - np.eye(2))) <= 1e-6
