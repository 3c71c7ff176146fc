"""The forms of the PSOD kernel (points, column strips; V, psi0 and the absorber in
shared memory or not) against the oracle on the sizes at their borders; |dC|, |dpsi|
<= 1e-10 (some roundings of 1.1e-16 per point and step on values of at most 1)."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu


def start(np_, seed):
    rng = np.random.default_rng(seed)
    axes = [np.linspace(-3.0, 3.0, n) if n > 1 else np.zeros(1) for n in np_]
    g = np.meshgrid(*axes, indexing="ij")
    v = sum(0.1 * x ** 2 for x in g)
    psi = np.exp(-sum((x - rng.uniform(-1, 1)) ** 2 for x in g) + 1.5j * g[0])
    shm = [1.0 / (24.0 * 1800.0 * (6.0 / max(n - 1, 1)) ** 2) for n in np_]
    psi = (psi / np.linalg.norm(psi)).ravel(order="F")
    mask = np.exp(-0.01 * np.maximum(g[0] - 2.0, 0.0) ** 2).ravel(order="F")
    return v.ravel(order="F"), psi, shm, mask


def plain(np_, shm, dt_au, v, psi, nsteps, mask):
    """psod.f on float64 arrays: Euler, midpoint, then steps of 2 dt."""
    def h(x):
        x = x.reshape(np_, order="F")
        out = (30.0 * sum(shm) + v.reshape(np_, order="F")) * x
        for ax, s in enumerate(shm):
            pad = [(2, 2) if i == ax else (0, 0) for i in range(len(np_))]
            p, n = np.pad(x, pad), x.shape[ax]
            take = lambda o: np.take(p, range(2 + o, 2 + o + n), axis=ax)
            out = out + s * (take(-2) + take(2) - 16.0 * (take(-1) + take(1)))
        return out.ravel(order="F")

    w = 1.0 if mask is None else mask
    cst = 2.0 * dt_au
    c = [np.vdot(psi, psi)]
    half = w * (psi - 1j * 0.25 * cst * h(psi))
    old, new = psi, w * (psi - 1j * 0.5 * cst * h(half))
    c.append(np.vdot(psi, new))
    for _ in range(nsteps - 1):
        old, new = new, w * (old - 1j * cst * h(new))
        c.append(np.vdot(psi, new))
    return np.array(c), new


SIZES = [[1], [31], [4000], [40000], [90001], [100, 100], [64, 1000], [63, 1000], [257, 300],
         [3, 20000], [400, 300], [1023, 769], [2100, 2000], [12, 13, 14], [50, 51, 52]]


@pytest.mark.parametrize("absorb", [False, True])
@pytest.mark.parametrize("np_", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_forms(np_, absorb):
    v, psi, shm, mask = start(np_, len(np_) + np_[0])
    dt_au = 0.2 / (64.0 * sum(shm) + v.max())
    nsteps = 6
    g = E.PsodGrid(np_, shm, dt_au * N.SHFS, absorb=N.ABS_SMOOTHW if absorb else N.ABS_NONE)
    c_ref, ref = plain(np_, shm, dt_au, v, psi, nsteps, mask if absorb else None)
    g.load(v, psi, vabc=mask if absorb else None)
    for ctas in (0, 7, 2) if np.prod(np_) > 7 * 256 else (0,):  # 256 points fill a CTA
        g.set_ctas(ctas)
        g.run(nsteps)
        c, out = g.results()
        assert np.max(np.abs(c - c_ref)) <= 1e-10
        assert np.max(np.abs(out - ref)) <= 1e-10
    # the same run in pieces
    g.set_ctas(0)
    g.run(2)
    c2, _ = g.results()
    g.advance(1)
    c3, _ = g.results()
    g.advance(nsteps - 3)
    c6, out = g.results()
    assert np.max(np.abs(np.concatenate([c2, c3[1:], c6[1:]]) - c_ref)) <= 1e-10
    assert np.max(np.abs(out - ref)) <= 1e-10
    g.close()
