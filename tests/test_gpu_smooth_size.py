"""1D packets of even sizes with prime factors up to 13 (espec_b200/csrc/
spo1d_smooth.cu): every radix of 2..16 as first, middle and last stage, two to
five stages, one thread to several butterflies per thread, next to a size with a
larger prime factor (the general path) in the same batch; the in-place defect;
runs cut into segments.  Against the oracle's restatement of spofft.f at the bar
of the register kernels, |dC(t)| and |d psi| <= 1e-10."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as NAT
from espec_b200 import workloads as W

from test_gpu_spo1d import gpu_batch, oracle_batch, random_packets

pytestmark = pytest.mark.gpu

SIZES = [4, 6, 8, 10, 12, 14, 16, 18, 20, 22, 24, 26, 28, 30, 32, 36, 44, 52, 60, 64, 66, 78, 90,
         98, 100, 110, 126, 128, 130, 144, 150, 168, 182, 196, 210, 220, 242, 260, 286, 338, 352,
         416, 450, 560, 640, 702, 900, 1144, 1500, 1694, 2000, 2310, 3000, 4032, 7200, 34]


@pytest.mark.parametrize("quirk", [False, True])
def test_smooth_sizes_match_oracle(oracle, quirk):
    n, off, sh, sm, v, psi = random_packets(SIZES, seed=5)
    dt = (0.005 if quirk else 0.5) * W.SHFS
    if quirk:
        # the defect's step is not unitary: with dt E_max above 1 its state grows
        # (to |psi| = 92 at 7200 points here) and so does every rounding of it
        ok = 0.005 * (np.pi / sh) ** 2 / (2.0 * sm) < 1.0
        pick = np.concatenate([np.arange(off[k], off[k + 1]) for k in np.nonzero(ok)[0]])
        n, sh, sm, v, psi = n[ok], sh[ok], sm[ok], v[pick], psi[pick]
        off = np.concatenate([[0], np.cumsum(n)])
    c_ref, p_ref = oracle_batch(oracle, n, off, sh, sm, v, psi, dt, 60,
                                quirks=oracle.Q_SPO_INPLACE if quirk else 0)
    c, p = gpu_batch(n, sh, sm, v, psi, dt, 60, "fp64", quirks=NAT.Q_SPO_INPLACE if quirk else 0)
    err = np.max(np.abs(c - c_ref), axis=1)
    assert np.max(err) <= 1e-10, dict(zip(n.tolist(), err))
    assert np.max(np.abs(p - p_ref)) <= 1e-10


def test_smooth_segments_and_zero_steps():
    n, off, sh, sm, v, psi = random_packets([250, 1500, 34], seed=6)
    b = E.SpoBatch(n, sh, sm, 0.5 * W.SHFS)
    b.load(v, psi)
    b.run(0)
    c0, p0 = b.results()
    assert np.allclose(p0, psi, rtol=0, atol=0)
    assert np.allclose(c0[:, 0], 1.0, atol=1e-14)
    b.run(30)
    c, p = b.results()
    b.run(13)
    ca, _ = b.results()
    b.advance(17)
    cb, pb = b.results()
    b.close()
    assert np.max(np.abs(ca - c[:, :14])) == 0.0
    assert np.max(np.abs(cb[:, 1:] - c[:, 14:])) <= 1e-13
    assert np.max(np.abs(pb - p)) <= 1e-13
