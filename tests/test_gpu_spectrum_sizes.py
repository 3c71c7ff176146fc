"""Spectrum stage at the sizes where its launch rule changes (1-3 passes, whole
transforms in shared memory with every remainder of the pass count, several
packets per CTA with a ragged last CTA, two and more groups above 2^13 points)
against numpy's FFT of the same formulas.  Bound: 64 eps log2 N of the
spectrum's largest value, for the mf stages' rounding and the factors'."""
import numpy as np
import pytest
import torch

from espec_b200 import spectrum as S

pytestmark = pytest.mark.gpu


def reference(c, mf, dt, tf, assemble, tal, de, window, wp):
    n, mc = 1 << mf, 1 << (mf - 1)
    j = np.arange(n)
    if assemble:
        x = np.empty((len(c), n), complex)
        x[:, 0] = np.conj(c[:, mc - 1])
        x[:, 1:mc + 1] = np.conj(c[:, mc - 1::-1])
        x[:, mc + 1:] = c[:, 1:mc]
    else:
        x = c[:, :n].copy()
    t = -tf + j * dt
    if tal is not None:
        x = x * np.exp(-1j * de * 1.5192676 * t - np.abs(t) * tal * 1.5192676)
    if window:
        x = x * np.exp(-t * t / ((n * dt) / np.log(1.0 / wp)) ** 2)
    return np.fft.ifft(np.roll(x, mc, axis=1), axis=1)


@pytest.mark.parametrize("mf", [1, 2, 3, 4, 5, 6, 7, 8, 11, 12, 13, 14, 15, 17])
@pytest.mark.parametrize("assemble", [True, False])
def test_spectrum_sizes(mf, assemble):
    rng = np.random.default_rng(mf)
    n = 1 << mf
    for npk, tal, window in ((1, None, None), (3, 0.02, None), (37, 0.01, "SG")):
        if mf > 14 and npk > 3:
            npk = 2
        ld = (n // 2 if assemble else n) + 3
        c = rng.standard_normal((npk, ld)) + 1j * rng.standard_normal((npk, ld))
        dt, de = 0.01, 1.3
        got = S.spectra(torch.from_numpy(c).cuda(), mf, dt, n // 2 * dt, assemble=assemble,
                        tal=tal, de=de, window=window).cpu().numpy()
        ref = reference(c, mf, dt, n // 2 * dt, assemble, tal, de, window, 1e-3)
        tol = 64 * np.finfo(float).eps * mf * np.max(np.abs(ref))
        assert np.max(np.abs(got - ref)) <= tol, (mf, npk)
