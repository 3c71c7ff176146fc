"""The order in which load() takes a wave function of several dimensions: batches and
FFT grids in C order, as they take the potential; finite-difference grids in Fortran
order (x first), potential and wave function alike.  A recorder stands in for the
native library."""
import ctypes as C

import numpy as np
import pytest

import espec_b200 as E
from espec_b200 import _native as N


class Recorder:
    def __init__(self, n):
        self.n = n

    def _copy(self, p, count):
        return np.array((C.c_double * count).from_address(p)) if p else None

    def _load(self, h, vpot, vabc, re, im, where, stream):
        self.v, self.ab = self._copy(vpot, self.n), self._copy(vabc, self.n)
        if where & N.MEM_INTERLEAVED:
            self.psi = self._copy(re, 2 * self.n).view(complex)
        else:
            im = self._copy(im, self.n)
            self.psi = self._copy(re, self.n) + 1j * (np.zeros(self.n) if im is None else im)
        return N.OK

    espec_spo_load = espec_grid_load = espec_spond_load = _load


CLASSES = {E.SpoBatch: "C", E.SodBatch: "C", E.SpoGrid: "C", E.SodGrid: "C", E.SilGrid: "F",
           E.PsodGrid: "F"}


@pytest.mark.parametrize("layout", ["c", "fortran", "strided"])
@pytest.mark.parametrize("shape", [(24,), (4, 6), (2, 3, 4)], ids=str)
@pytest.mark.parametrize("kind", ["complex", "complex64", "real"])
@pytest.mark.parametrize("cls", list(CLASSES), ids=lambda c: c.__name__)
def test_order(monkeypatch, cls, kind, shape, layout):
    rng = np.random.default_rng(7)
    v, ab, psi = rng.random(shape), rng.random(shape), rng.random(shape)
    if kind != "real":
        psi = (psi + 1j * rng.random(shape)).astype(complex if kind == "complex" else "c8")
    if layout == "fortran":
        psi = np.asfortranarray(psi)
    elif layout == "strided":
        psi = np.repeat(psi, 2, axis=-1)[..., ::2]
    plan = cls.__new__(cls)
    plan._h = None
    lib = Recorder(v.size)
    monkeypatch.setattr(N, "load", lambda: lib)
    plan.load(v, psi, ab)
    order = CLASSES[cls]
    assert np.array_equal(lib.psi, psi.ravel(order=order))
    assert np.array_equal(lib.v, v.ravel(order=order))
    assert np.array_equal(lib.ab, ab.ravel(order=order))
