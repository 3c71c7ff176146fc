"""Interleaved arrays of grid plans with ESPEC_MEM_HOST_ASYNC (page-locked memory, the
stream synchronised by the caller) as with ESPEC_MEM_HOST; the calls for the previous
state, which have no interleaved form, refuse it before anything is launched."""
import numpy as np
import pytest
import torch

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu
GRIDS = {
    "sil": (lambda: E.SilGrid([30, 20], [1e-3] * 2, 0.01, 6), "grid", 600),
    "psod": (lambda: E.PsodGrid([700], [1e-3], 0.001), "grid", 700),
}


@pytest.mark.parametrize("kind", list(GRIDS))
def test_host_async(kind):
    make, name, n = GRIDS[kind]
    lib, st = N.load(), torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(n)
    v = torch.from_numpy(0.1 * rng.random(n)).pin_memory()
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    z = torch.from_numpy(z / np.linalg.norm(z)).pin_memory()
    got = []
    for where in (N.MEM_HOST, N.MEM_HOST_ASYNC):
        where |= N.MEM_INTERLEAVED
        p = make()
        N.check(lib.espec_grid_load(p._h, v.data_ptr(), None, z.data_ptr(), None, where, st),
                "load")
        p.run(5, stream=st)
        c = torch.zeros(6, dtype=torch.complex128).pin_memory()
        psi = torch.zeros(n, dtype=torch.complex128).pin_memory()
        for out in ((c, None), (None, psi)):
            N.check(lib.espec_grid_results(p._h, *[x if x is None else x.data_ptr() for x in
                                                   (out[0], None, out[1], None)], where, st),
                    "results")
        torch.cuda.synchronize()
        got.append((c.numpy(), psi.numpy()))
        p.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert abs(got[0][0][0] - 1) < 1e-12


@pytest.mark.parametrize("make,call", [
    (lambda: E.SodBatch([64], [0.05], [1836.0], 1e-4), "espec_prop_previous"),
    (lambda: E.SodGrid([32, 32], [0.3] * 2, [1836.0] * 2, 1e-3), "espec_spond_previous"),
    (lambda: E.PsodGrid([700], [1e-3], 0.001), "espec_grid_previous")],
    ids=["batch", "fft", "fd"])
def test_previous_refuses(make, call):
    p = make()
    n = p.total if hasattr(p, "total") else p.n
    p.load(np.zeros(n), np.ones(n) / np.sqrt(n) + 0j)
    p.run(3)
    out = np.zeros(2 * n)
    rc = getattr(N.load(), call)(p._h, out.ctypes.data, None, N.MEM_HOST | N.MEM_INTERLEAVED, None)
    assert rc == -1 and not out.any()
    assert np.isfinite(p.previous()).all()
    p.close()
