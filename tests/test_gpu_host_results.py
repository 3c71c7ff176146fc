"""Results of a plan into separate host arrays when C(t) fits the plan's small
page-locked block and psi does not, on plans whose load left no staging block (complex
or device arrays): the values of the interleaved results, bit for bit."""
import numpy as np
import pytest
import torch

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu


def plan_of(kind):
    if kind == "batch":
        k = 8
        return E.SpoBatch([1024] * k, [0.05] * k, [1836.0] * k, 0.01), "spo", 8192, k, 100
    if kind == "sod_batch":
        return E.SodBatch([2048] * 4, [0.05] * 4, [1836.0] * 4, 1e-4), "prop", 8192, 4, 10
    if kind == "spo2d":
        return E.SpoGrid([256, 256], [0.05] * 2, [1836.0] * 2, 0.01), "spond", 65536, 1, 20
    return E.SodGrid([64, 64], [0.3] * 2, [1836.0] * 2, 1e-3), "spond", 4096, 1, 12


@pytest.mark.parametrize("source", ["complex", "device"])
@pytest.mark.parametrize("kind", ["batch", "sod_batch", "spo2d", "sod2d"])
def test_small_c_large_psi(kind, source):
    plan, name, n, npk, steps = plan_of(kind)
    lib, st = N.load(), torch.cuda.current_stream().cuda_stream
    family = "spo" if name == "prop" else name
    load, res = getattr(lib, f"espec_{family}_load"), getattr(lib, f"espec_{family}_results")
    rng = np.random.default_rng(n)
    v = 0.1 * rng.random(n)
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    z /= np.linalg.norm(z)
    if source == "complex":
        N.check(load(plan._h, N.ptr(v), None, N.ptr(z), None, N.MEM_HOST | N.MEM_INTERLEAVED, st),
                "load")
    else:
        d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (v, z.real, z.imag)]
        N.check(load(plan._h, N.ptr(d[0]), None, N.ptr(d[1]), N.ptr(d[2]), N.MEM_DEVICE, st),
                "load")
    plan.run(steps, stream=st)
    nc = npk * (steps + 1)
    a = [np.zeros(nc), np.zeros(nc), np.zeros(n), np.zeros(n)]
    N.check(res(plan._h, *[N.ptr(x) for x in a], N.MEM_HOST, st), "results")
    if kind.startswith("sod"):  # a second result of its own, from the block that stayed
        prev = getattr(lib, f"espec_{name}_previous")
        b = [np.zeros(n), np.zeros(n)]
        N.check(prev(plan._h, N.ptr(b[0]), N.ptr(b[1]), N.MEM_HOST, st), "previous")
        assert np.array_equal(b[0] + 1j * b[1], plan.previous())
    c, psi = plan.results(stream=st)
    assert np.isfinite(psi).all() and abs(c.reshape(npk, -1)[0, 0]) > 0
    assert np.array_equal(a[0] + 1j * a[1], c.ravel())
    assert np.array_equal(a[2] + 1j * a[3], psi)
    plan.close()
