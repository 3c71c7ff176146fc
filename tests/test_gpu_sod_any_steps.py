"""Second-order differences on packets of sizes outside the register plans, the first
steps one by one: 2 to 5 steps against the oracle, and runs continued after each of
them against one run, bit for bit.  Sizes of 2, 3 and 5 and sizes with a larger prime
factor run two forms of the kernel.  1e-10 is the tests' bound for FP64."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import workloads as W
from test_gpu_sod import oracle_sod, packet

pytestmark = pytest.mark.gpu
STEPS = 5


@pytest.mark.parametrize("n", [60, 90, 250, 242, 1022])
def test_first_steps(oracle, n):
    _, sh, sm, v, psi = packet(n, n)
    dt = 0.002 * W.SHFS
    b = E.SodBatch([n], [sh], [sm], dt)
    b.load(v, psi)
    states = []
    for k in range(STEPS + 1):
        b.run(k)
        c, u = b.results()
        states.append((u, b.previous(), c[0]))
    assert np.all(states[0][0] == psi)
    for k in range(1, STEPS):
        r = oracle_sod(oracle, n, sh, sm, v, psi, dt, k)
        u, _, c = states[r["nc"] - 1]  # its loop takes up to a step more than k
        assert np.max(np.abs(c - r["c"])) <= 1e-10
        assert np.max(np.abs(u - (r["u"] + 1j * r["v"]))) <= 1e-10
    assert np.all(states[1][1] == psi)  # psi(t - dt) after one step
    for k in range(1, STEPS + 1):
        assert k == 1 or np.all(states[k][1] == states[k - 1][0])
        b.run(k)
        b.advance(STEPS - k)
        assert np.all(b.results()[1] == states[STEPS][0])
        assert np.all(b.previous() == states[STEPS][1])
