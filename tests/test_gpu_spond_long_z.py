"""3D FFT grids with z lines of 512 points (separate passes) and the longest ones below
(fused planes) against the oracle: SPO, SOD and the energies, |dC|, |dpsi| <= 1e-10 (some
hundred roundings of 1.1e-16 per step on values of at most 1, 6 steps)."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as NAT

from test_gpu_spond import gpu_sod, gpu_spo, oracle_sod, oracle_spo, packet

pytestmark = pytest.mark.gpu
SHAPES = [[32, 32, 512], [64, 32, 512], [32, 64, 512], [32, 32, 256]]


@pytest.mark.parametrize("np_", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_long_z(oracle, np_):
    v, psi, sh, sm, _ = packet(np_, 17)
    dt = 0.002 * NAT.SHFS
    ref, nst = oracle_spo(oracle, np_, sh, sm, dt, 5, v, psi)
    c, out = gpu_spo(np_, sh, sm, dt, v, psi, nst)
    assert np.max(np.abs(c - ref["c"])) <= 1e-10
    assert np.max(np.abs(out - (ref["u"] + 1j * ref["v"]))) <= 1e-10
    dt = 2e-5 * NAT.SHFS
    ref = oracle_sod(oracle, np_, sh, sm, dt, 5, v, psi)
    c, out, prev = gpu_sod(np_, sh, sm, dt, v, psi, ref["nc"] - 1)
    assert np.max(np.abs(c - ref["c"])) <= 1e-10
    assert np.max(np.abs(out - (ref["u"] + 1j * ref["v"]))) <= 1e-10
    assert np.max(np.abs(prev - (ref["u_prev"] + 1j * ref["v_prev"]))) <= 1e-10


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("np_", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_energy(np_, precision):
    """Mean energy of psi(0), both in x space and by the axis tables' sum in k space."""
    v, psi, sh, sm, _ = packet(np_, 18)
    g = E.SpoGrid(np_, sh, sm, 0.002 * NAT.SHFS, precision=precision)
    g.load(v, psi)
    e, norm = g.energies()
    g.close()
    shape = np_[::-1]
    k2 = np.zeros(shape)
    for ax, n in enumerate(np_):
        tc = (np.fft.fftfreq(n) * n * 6.283185307 / (n * sh[ax])) ** 2 / (2 * sm[ax])
        k2 = k2 + tc.reshape([-1 if i == 2 - ax else 1 for i in range(3)])
    x = psi.reshape(shape)
    want = np.sum(v.reshape(shape) * np.abs(x) ** 2) + \
        np.sum(k2 * np.abs(np.fft.fftn(x)) ** 2) / x.size
    assert abs(norm - 1.0) <= 1e-13 and abs(e - want) <= 1e-11 * abs(want)
