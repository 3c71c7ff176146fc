"""A program may overwrite its complex wave function as soon as load() has returned, also
where the array is page-locked and the stream is busy."""
import numpy as np
import pytest
import torch

import espec_b200 as E

pytestmark = pytest.mark.gpu
PLANS = {
    "batch": lambda: E.SpoBatch([1024] * 64, [0.05] * 64, [1836.0] * 64, 0.01),
    "mixed_sizes": lambda: E.SpoBatch([512, 1000, 64], [0.05] * 3, [1836.0] * 3, 0.01),
    "spo2d": lambda: E.SpoGrid([128, 128], [0.05] * 2, [1836.0] * 2, 0.01),
    "sod3d": lambda: E.SodGrid([32, 32, 32], [0.3] * 3, [1836.0] * 3, 1e-3),
    "sil": lambda: E.SilGrid([60, 50], [1e-3] * 2, 0.01, 5),
    "psod": lambda: E.PsodGrid([256, 256], [1e-3] * 2, 0.001),
}
SIZE = {"batch": 65536, "mixed_sizes": 1576, "spo2d": 16384, "sod3d": 32768, "sil": 3000,
        "psod": 65536}


@pytest.mark.parametrize("kind", list(PLANS))
def test_overwritten_after_load(kind):
    n = SIZE[kind]
    rng = np.random.default_rng(n)
    v = torch.from_numpy(0.05 * rng.random(n)).pin_memory().numpy()
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    z /= np.linalg.norm(z)
    p = PLANS[kind]()
    p.load(v, z)
    p.run(3)
    want = p.results()
    kept = torch.from_numpy(z.copy()).pin_memory()
    x = kept.numpy()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        p.load(v, x, stream=st.cuda_stream)
        x[:] = 0.0
        p.run(3, stream=st.cuda_stream)
        got = p.results(stream=st.cuda_stream)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    p.close()
