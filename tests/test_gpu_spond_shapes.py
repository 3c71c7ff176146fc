"""The forms of the 2D/3D cooperative kernel against the oracle: every line
length, both CTA sizes, fused xy planes and separate passes, staged and direct
kinetic tiles; C(t) and psi within 1e-10 (some hundred roundings of 1.1e-16 per
step on values of at most 1, 6 steps), the mixed form within FP32 rounding."""
import numpy as np
import pytest

from espec_b200 import _native as NAT

from test_gpu_spond import gpu_sod, gpu_spo, oracle_sod, oracle_spo, packet
import espec_b200 as E

pytestmark = pytest.mark.gpu

SHAPES = [[32, 32], [512, 32], [32, 512], [256, 128], [128, 256], [64, 512],  # 2D
          [32, 32, 32], [32, 32, 512], [512, 32, 32], [32, 256, 32],         # 3D
          [32, 32, 64], [64, 32, 128], [32, 64, 256], [256, 32, 64],
          [128, 64, 64], [64, 64, 128]]
DT = 0.002 * NAT.SHFS


@pytest.mark.parametrize("np_", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_spo_forms(oracle, np_):
    v, psi, sh, sm, _ = packet(np_, 7)
    ref, nst = oracle_spo(oracle, np_, sh, sm, DT, 5, v, psi)
    c, out = gpu_spo(np_, sh, sm, DT, v, psi, nst)
    want = ref["u"] + 1j * ref["v"]
    assert np.max(np.abs(c - ref["c"])) <= 1e-10
    assert np.max(np.abs(out - want)) <= 1e-10
    # FP32 data: a transform rounds to a few 6e-8 of the 2-norm (1 here) per pass
    c, out = gpu_spo(np_, sh, sm, DT, v, psi, nst, precision="mixed")
    assert np.max(np.abs(c - ref["c"])) <= 1e-5
    assert np.linalg.norm(out - want) <= 1e-5


@pytest.mark.parametrize("np_", [[32, 512], [256, 128], [32, 32, 32], [64, 32, 128]],
                         ids=lambda s: "x".join(map(str, s)))
def test_sod_forms(oracle, np_):
    v, psi, sh, sm, _ = packet(np_, 8)
    dt = 2e-5 * NAT.SHFS
    ref = oracle_sod(oracle, np_, sh, sm, dt, 5, v, psi)
    c, out, prev = gpu_sod(np_, sh, sm, dt, v, psi, ref["nc"] - 1)
    assert np.max(np.abs(c - ref["c"])) <= 1e-10
    assert np.max(np.abs(out - (ref["u"] + 1j * ref["v"]))) <= 1e-10
    assert np.max(np.abs(prev - (ref["u_prev"] + 1j * ref["v_prev"]))) <= 1e-10


@pytest.mark.parametrize("cls,np_", [(E.SpoGrid, [64, 64]), (E.SpoGrid, [32, 32, 64]),
                                     (E.SodGrid, [64, 64]), (E.SodGrid, [32, 32, 64])])
def test_run_in_pieces(cls, np_):
    """run(4) + advance(1) + advance(2) against run(7)."""
    v, psi, sh, sm, _ = packet(np_, 9)
    dt = 2e-5 * NAT.SHFS
    g = cls(np_, sh, sm, dt)
    g.load(v, psi)
    g.run(7)
    c7, p7 = g.results()
    g.run(4)
    c4, _ = g.results()
    g.advance(1)
    c1, _ = g.results()
    g.advance(2)
    c2, p2 = g.results()
    g.close()
    c = np.concatenate([c4, c1[1:], c2[1:]])
    # the pieces round the merged half-steps apart: a few 1.1e-16 per step
    assert np.max(np.abs(c - c7)) <= 1e-12
    assert np.max(np.abs(p2 - p7)) <= 1e-12
