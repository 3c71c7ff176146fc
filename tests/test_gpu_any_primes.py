"""1D packets whose size has prime factors of 7 and more (prime_stage of
espec_b200/csrc/spo1d_any.cu): SPO, SOD with the FFT and the energies against the
oracle at 1e-10, the bar of the other sizes; with the table of the prime's roots in
shared memory, and (7246 = 2 x 3623, SOD 3622 = 2 x 1811) without room for it."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import workloads as W

from test_gpu_sod import oracle_sod, packet
from test_gpu_spo1d import gpu_batch, oracle_batch, random_packets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,steps", [
    ([34, 38, 62, 194], 60), ([578, 646, 1102, 442], 60), ([1322, 1326, 1794], 40),
    ([2 * 1811], 20), ([2 * 3623], 10)], ids=str)
def test_spo_prime_factors(oracle, sizes, steps):
    n, off, sh, sm, v, psi = random_packets(sizes, seed=sizes[0])
    dt = 0.5 * W.SHFS
    c_ref, p_ref = oracle_batch(oracle, n, off, sh, sm, v, psi, dt, steps)
    c, p = gpu_batch(n, sh, sm, v, psi, dt, steps, "fp64")
    assert np.max(np.abs(c - c_ref)) <= 1e-10
    assert np.max(np.abs(p - p_ref)) <= 1e-10


@pytest.mark.parametrize("n", [98, 242, 286, 1022, 3622])
def test_sod_prime_factors(oracle, n):
    x, sh, sm, v, psi = packet(n, n)
    # SOD is stable for dt E_max < 1
    dt = 0.1 / (0.5 * (np.pi / sh) ** 2 / sm + np.max(np.abs(v))) * W.SHFS
    r = oracle_sod(oracle, n, sh, sm, v, psi, dt, 6)
    b = E.SodBatch([n], [sh], [sm], dt)
    b.load(v, psi)
    b.run(r["nc"] - 1)
    c, out = b.results()
    b.close()
    assert np.max(np.abs(c[0] - r["c"])) <= 1e-10
    assert np.max(np.abs(out - (r["u"] + 1j * r["v"]))) <= 1e-10


@pytest.mark.parametrize("n", [34, 1322, 7246])
def test_energies_prime_factors(oracle, n):
    n, off, sh, sm, v, psi = random_packets([n], seed=n)
    b = E.SpoBatch(n, sh, sm, 0.1 * W.SHFS, precision="fp64")
    b.load(v, psi)
    e, nrm = b.energies()
    b.close()
    tc, bb = oracle.digt([int(n[0])], [sh[0]], [sm[0]])
    e_ref = oracle.efft4([int(n[0])], psi, np.zeros(int(n[0])), tc, v, bb)
    assert abs(e[0] - e_ref) <= 1e-12 * max(1.0, abs(e_ref))
    assert abs(nrm[0] - np.sum(psi ** 2)) <= 1e-12
