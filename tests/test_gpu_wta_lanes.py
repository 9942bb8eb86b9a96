"""The winner-take-all over every number of single loads per lane: ties,
infinities and NaN as in test_gpu_right_view.py."""
import pytest

from test_gpu_right_view import test_winner_take_all as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [33, 63, 64, 65, 96, 97, 127, 128, 129, 255])
def test_rows_in_lanes(gpu, D):
    for off in (0, 1):
        _check(gpu, D, off)
