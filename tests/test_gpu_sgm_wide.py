"""The SGM scan with 32 disparities per lane, whose rows are padded in shared
memory, over vectors of 4, 2 and 1: the recursion of test_gpu_sgm_lanes.py."""
import pytest

from test_gpu_sgm_lanes import test_sgm_equals_float32_model as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [769, 770, 772, 897, 1000, 1022, 1023])
@pytest.mark.parametrize("direction", [-1, 1])
def test_rows_of_769_to_1024(gpu, D, direction):
    _check(gpu, D, direction)
