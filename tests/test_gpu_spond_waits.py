"""A grid barrier of the 2D/3D FFT kernels that gives up (a launch whose arrival count
starts one short, with a short limit): results, the previous state and the energies
report it, also after a continued run; a new load, a new run and energies of their own
are not touched by it."""
import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    lib = N.load()
    assert lib.espec_set_wait_limit(1 << 12) == 0
    yield lib
    lib.espec_selftest_short_arrivals(0)
    lib.espec_set_wait_limit(0)


def make(cls, shape):
    rng = np.random.default_rng(5)
    n = int(np.prod(shape))
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    g = cls(shape, [0.3] * len(shape), [1836.0] * len(shape), 1e-3)
    return g, (0.1 * rng.random(n), z / np.linalg.norm(z))


@pytest.mark.parametrize("shape", [[64, 64], [32, 32, 64]], ids=str)
@pytest.mark.parametrize("cls", [E.SpoGrid, E.SodGrid], ids=lambda c: c.__name__)
def test_run_gives_up(cls, shape, lib):
    g, data = make(cls, shape)
    g.load(*data)
    e0 = g.energies()
    g.run(4)
    ref = g.results(), g.energies()
    lib.espec_selftest_short_arrivals(1)
    g.run(4)
    for _ in range(2):
        for call in (g.results, g.energies, *([g.previous] if cls is E.SodGrid else [])):
            with pytest.raises(E.EspecError, match="timed out"):
                call()
        g.advance(3)  # from the spoilt state: still reported
    g.load(*data)
    assert g.energies() == e0
    g.run(4)
    (c, psi), e = g.results(), g.energies()
    assert np.array_equal(c, ref[0][0]) and np.array_equal(psi, ref[0][1]) and e == ref[1]
    g.close()


def test_energies_give_up(lib):
    g, data = make(E.SpoGrid, [64, 64])
    g.load(*data)
    g.run(4)
    ref, e = g.results(), g.energies()
    lib.espec_selftest_short_arrivals(1)
    with pytest.raises(E.EspecError, match="timed out"):
        g.energies()
    c, psi = g.results()
    assert np.array_equal(c, ref[0]) and np.array_equal(psi, ref[1]) and g.energies() == e
    g.close()
