"""Places a CTA of the PSOD kernel needs for the constants of its points: the points of
a brute-force walk, and no wrap at the largest grids (64 x 2^24 points in one band)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include <cstdio>
#include <cstdlib>
#include "sil.cuh"
int main(int argc, char** v) {
  std::printf("%ld\\n", espec::psod_places(atoi(v[1]), atol(v[2]), atoi(v[3]), atoi(v[4])));
}
"""


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    d = tmp_path_factory.mktemp("places")
    (d / "p.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "espec_b200", "csrc"), str(d / "p.cpp"), "-o",
                    str(d / "p")], check=True)
    return lambda *a: int(subprocess.run([str(d / "p"), *map(str, a)], check=True,
                                         capture_output=True, text=True).stdout)


@pytest.mark.parametrize("nx,ny,nblocks", [(64, 600, 148), (64, 601, 300), (300, 7, 6),
                                           (1023, 769, 296), (256, 9, 5), (257, 100, 98)])
def test_bands(places, nx, ny, nblocks):
    strips = -(-nx // 256)
    bands = nblocks // strips
    rows = -(-ny // bands)
    most = max(min((b + 1) * rows, ny) - min(b * rows, ny) for b in range(bands))
    assert places(strips, nx * ny, ny, nblocks) == most * 256


@pytest.mark.parametrize("n,nblocks", [(1, 1), (1000, 7), (40 ** 3, 148), (2 ** 30, 1)])
def test_ranges(places, n, nblocks):
    assert places(0, n, 1, nblocks) == -(-n // nblocks)


@pytest.mark.parametrize("nx,ny", [(64, 2 ** 24), (128, 2 ** 23), (100, 10737418)])
def test_largest(places, nx, ny):
    assert places(1, nx * ny, ny, 1) == ny * 256
