"""The page-locked blocks that plans share for small results: more plans alive than
blocks, plans made and closed over and over, several threads -- every plan reads its own
values, those of the interleaved results, which take no block."""
import threading

import numpy as np
import pytest

import espec_b200 as E

pytestmark = pytest.mark.gpu


def plan(k):
    n = 32 + 2 * (k % 50)
    p = E.SpoBatch([n], [0.05], [1836.0], 0.01)
    rng = np.random.default_rng(k)
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    p.load(0.1 * rng.random(n), z / np.linalg.norm(z))
    p.run(3 + k % 4)
    return p


def check(p):
    out = [np.zeros(m) for m in (p.nsteps + 1, p.nsteps + 1, p.total, p.total)]
    p.results_into(*out)
    e, norm = p.energies()
    c, psi = p.results()
    assert np.array_equal(out[0] + 1j * out[1], c.ravel())
    assert np.array_equal(out[2] + 1j * out[3], psi)
    assert abs(norm[0] - np.sum(np.abs(psi) ** 2)) < 1e-14 * len(psi) and np.isfinite(e).all()


def test_many_plans():
    alive = [plan(k) for k in range(40)]
    for _ in range(4):  # past the first requests, which are copied
        for p in alive:
            check(p)
    for p in alive[::2]:
        p.close()
    late = [plan(k) for k in range(100, 130)]
    for p in alive[1::2] + late:
        check(p)
        p.close()


def test_threads():
    failed = []

    def work(k):
        try:
            for j in range(30):
                p = plan(1000 * k + j)
                check(p)
                check(p)
                p.close()
        except Exception as e:  # reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]
