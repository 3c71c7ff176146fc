"""Interleaved (re, im) arrays in the load and results calls of every plan kind,
from host and device memory, against separate arrays: the same bits.  Batches of one
packet size and of several, results inside and beyond the small page-locked space."""
import numpy as np
import pytest
import torch

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu
PI = N.MEM_INTERLEAVED


def plans():
    def batch(sizes):
        n = np.array(sizes)
        return (E.SpoBatch(n, np.full(len(n), 0.05), np.full(len(n), 1836.0), 0.01), "spo",
                int(n.sum()), len(n))
    return {
        "one_size": lambda: batch([256]), "many_equal": lambda: batch([512] * 9),
        "mixed_sizes": lambda: batch([64, 100, 384, 1024]),
        "spo2d": lambda: (E.SpoGrid([32, 64], [0.05] * 2, [1836.0] * 2, 0.01), "spond", 2048, 1),
        "sod3d": lambda: (E.SodGrid([32, 32, 32], [0.3] * 3, [1836.0] * 3, 0.001), "spond",
                          32768, 1),
        "sil": lambda: (E.SilGrid([30, 20], [1e-3] * 2, 0.01, 6), "grid", 600, 1),
        "psod": lambda: (E.PsodGrid([700], [1e-3], 0.001), "grid", 700, 1),
    }


@pytest.mark.parametrize("kind", list(plans()))
def test_interleaved(kind):
    plan, name, n, npk = plans()[kind]()
    lib, st = N.load(), torch.cuda.current_stream().cuda_stream
    load, res = getattr(lib, f"espec_{name}_load"), getattr(lib, f"espec_{name}_results")
    rng = np.random.default_rng(n)
    v = 0.1 * rng.random(n)
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    z /= np.linalg.norm(z)
    parts = [np.ascontiguousarray(z.real), np.ascontiguousarray(z.imag)]
    dv, dz = torch.from_numpy(v).cuda(), torch.from_numpy(z).cuda()
    dparts = [torch.from_numpy(p).cuda() for p in parts]
    out = []
    for steps in (3, 40):
        nc = npk * (steps + 1)
        for src in ("host", "device"):
            where = N.MEM_HOST if src == "host" else N.MEM_DEVICE
            for pairs in (False, True):
                pot = N.ptr(v if src == "host" else dv)
                re, im = ([N.ptr(z if src == "host" else dz), None] if pairs else
                          [N.ptr(p) for p in (parts if src == "host" else dparts)])
                N.check(load(plan._h, pot, None, re, im, where | (PI if pairs else 0), st), "load")
                plan.run(steps, stream=st)
                new = (lambda k: np.zeros(k)) if src == "host" else (
                    lambda k: torch.zeros(k, dtype=torch.float64, device="cuda"))
                if pairs:
                    c, p = new(2 * nc), new(2 * n)
                    N.check(res(plan._h, N.ptr(c), None, N.ptr(p), None, where | PI, st), "res")
                    torch.cuda.synchronize()
                    c, p = [np.asarray(x if src == "host" else x.cpu()).view(complex)
                            for x in (c, p)]
                else:
                    a = [new(nc), new(nc), new(n), new(n)]
                    N.check(res(plan._h, *[N.ptr(x) for x in a], where, st), "res")
                    torch.cuda.synchronize()
                    a = [np.asarray(x if src == "host" else x.cpu()) for x in a]
                    c, p = a[0] + 1j * a[1], a[2] + 1j * a[3]
                out.append((c, p))
        first = out[0]
        assert np.isfinite(first[0]).all() and abs(np.linalg.norm(first[1]) - 1) < 0.1
        for c, p in out[1:]:
            assert np.array_equal(c, first[0]) and np.array_equal(p, first[1])
        out = []
    plan.close()
