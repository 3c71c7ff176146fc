"""The eigensolver at the grid sizes where the points per thread change: 512 (one), 1024
(two) and a point more or less; checks and bounds of the small grids."""
import pytest

from test_gpu_eig_small import test_small as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_", [(7, 73), (16, 32), (19, 27), (25, 41)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_points_per_thread(np_):
    check(np_, 3)
