"""Spectra written over their own samples (spec = in), every kind of launch, and packets
whose samples lie further back in the spectra's memory: the values of the call with
separate buffers.  Bound: 64 eps log2 N of the spectrum's largest value, as two orders of
the same passes differ."""
import numpy as np
import pytest
import torch

from espec_b200 import _native as N

pytestmark = pytest.mark.gpu


def spectrum(c, ld, npk, mf, assemble, scaled, out):
    lib = N.load()
    work = torch.empty(lib.espec_spectrum_work_bytes(npk, mf) // 16, dtype=torch.complex128,
                       device="cuda")
    n = 1 << mf
    N.check(lib.espec_spectrum_dev(npk, mf, c.data_ptr(), ld, int(assemble), 0.01, n // 2 * 0.01,
                                   0.02 if scaled else -1.0, 1.3, int(scaled), 1e-3, 0,
                                   out.data_ptr(), work.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream), "espec_spectrum_dev")
    return out


@pytest.mark.parametrize("mf", [1, 3, 4, 5, 8, 12, 13, 14, 15, 17])
@pytest.mark.parametrize("scaled", [False, True])
def test_spectrum_in_place(mf, scaled):
    n, npk = 1 << mf, 5 if mf < 14 else 2
    rng = np.random.default_rng(mf)
    c = torch.from_numpy(rng.standard_normal((npk, n)) + 1j * rng.standard_normal((npk, n))).cuda()
    # samples as long as the spectra, and half as long and assembled
    for assemble, ld in ((False, n), (True, n // 2)):
        src = c.flatten()[:npk * ld].clone()
        ref = spectrum(src, ld, npk, mf, assemble, scaled, torch.empty_like(c)).cpu().numpy()
        tol = 64 * np.finfo(float).eps * mf * np.max(np.abs(ref))
        for off in sorted({0, npk * n - npk * ld}):
            buf = torch.zeros(npk * n, dtype=torch.complex128, device="cuda")
            buf[off:off + npk * ld] = src
            got = spectrum(buf[off:], ld, npk, mf, assemble, scaled, buf)
            err = np.max(np.abs(got.cpu().numpy().reshape(npk, n) - ref))
            assert err <= tol, (assemble, off)
