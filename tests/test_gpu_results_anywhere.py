"""Results asked for in host memory (ESPEC_MEM_HOST) whose destinations are device
pointers: the unified address space lets the copies take them, for small results as for
large ones."""
import numpy as np
import pytest
import torch

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("on_device", ["re", "im", "both"])
@pytest.mark.parametrize("n,steps", [(64, 3), (512, 40), (4096, 2)])
def test_device_destination(n, steps, on_device):
    p = E.SpoBatch([n], [0.05], [1836.0], 0.01)
    rng = np.random.default_rng(n)
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    p.load(0.1 * rng.random(n), z / np.linalg.norm(z))
    p.run(steps)
    c, psi = p.results()

    def place(k, part):
        if on_device in (part, "both"):
            return torch.zeros(k, dtype=torch.float64, device="cuda")
        return np.zeros(k)

    out = [place(k, part) for k in (steps + 1, n) for part in ("re", "im")]
    N.check(N.load().espec_spo_results(p._h, *[N.ptr(x) for x in out], N.MEM_HOST,
                                       torch.cuda.current_stream().cuda_stream), "results")
    cr, ci, pr, pi = [x if isinstance(x, np.ndarray) else x.cpu().numpy() for x in out]
    assert np.array_equal(cr + 1j * ci, c.ravel()) and np.array_equal(pr + 1j * pi, psi)
    p.close()
