"""The PSOD kernel's column strips and its points with the constants in shared memory
against the oracle, with what changes the arithmetic of a point: both absorbers, the
restart-copy defect, a pulse.  Strips with the constants in shared memory (400 x 300,
257 x 300, 72 x 700) and without (1300 x 1250), points in 1D, 2D (71 x 700) and 3D.  Some
roundings of 1.1e-16 per point and step on values of at most 1: |dC|, |dpsi| <= 1e-10."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as N
from espec_b200 import grid as GR

import golden_cases as G
from test_gpu_psod import packet

pytestmark = pytest.mark.gpu
SIZES = {"400x300": 1e-4, "257x300": 1e-4, "72x700": 1e-4, "71x700": 1e-4,
         "1300x1250": 1e-5, "90001": 2e-8, "50x51x52": 1e-3}


@pytest.mark.parametrize("extra", ["plain", "copy", "pulse"])
@pytest.mark.parametrize("absorb", [N.ABS_NONE, N.ABS_VOPTIC, N.ABS_SMOOTHW],
                         ids=["none", "voptic", "smoothw"])
@pytest.mark.parametrize("size", list(SIZES))
def test_point_arithmetic(oracle, size, absorb, extra):
    np_ = [int(k) for k in size.split("x")]
    v, psi, sh, grids = packet(np_, 11 + absorb)
    sm = [1000.0 + 400.0 * a for a in range(len(np_))]
    shm = [G.shm_of(m, h) for m, h in zip(sm, sh)]
    dt = SIZES[size] * N.SHFS
    assert SIZES[size] * (64.0 * sum(shm) + v.max()) < 1.0  # stable steps
    steps = 7
    vabc = None
    if absorb == N.ABS_VOPTIC:
        vabc = -0.05 * np.clip(grids[0] - 0.3, 0, None).ravel(order="F") ** 2
    elif absorb == N.ABS_SMOOTHW:
        vabc = np.where(grids[0] > 0.35, 0.97, 1.0).ravel(order="F")
    quirk = extra == "copy"
    p = oracle.make_prop(np_, dt, 0.0, steps * dt, sh, sm, lc=1, absorb=absorb, shm=shm,
                         quirks=oracle.Q_PSOD_COPY if quirk else 0)
    g = E.PsodGrid(np_, shm, dt, absorb=absorb, quirks=N.Q_PSOD_COPY if quirk else 0)
    g.load(v, psi, vabc=vabc)
    if extra == "pulse":
        dm = (0.8 * grids[0] + 0.3 * grids[0] ** 2).ravel(order="F")
        shape, par = N.PULSE_GAUS, (6e9, 0.08, 2.5, 0.0, 0.3)
        ef = GR.ppsod_field(shape, par, 0.0, steps * dt, dt)
        assert np.max(np.abs(ef)) > 1e-4
        ref = oracle.ppsod(p, v, dm, shape, par, np.real(psi), np.imag(psi), vabc=vabc)
        g.set_pulse(dm, ef)
    else:
        ref = oracle.psod(p, v, np.real(psi), np.imag(psi), vabc=vabc)
    g.run(ref["nc"] - 1)
    c, out = g.results()
    prev = g.previous()
    g.close()
    assert np.max(np.abs(c - ref["c"])) <= 1e-10
    assert np.max(np.abs(out - (ref["u"] + 1j * ref["v"]))) <= 1e-10
    assert np.max(np.abs(prev - (ref["u_prev"] + 1j * ref["v_prev"]))) <= 1e-10
