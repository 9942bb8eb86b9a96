"""The float64 and float32 matchers on both sides of the lines between the
general and the strip kernels, against the oracle: equal (float32: the
rounding of the float64 value)."""
import numpy as np
import pytest

from conftest import rand_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,D", [(17, 40, 3), (17, 40, 4), (13, 50, 5), (13, 50, 10), (19, 37, 11), (19, 37, 12),
                                   (14, 61, 13), (14, 61, 14), (250, 400, 5), (250, 400, 6), (180, 300, 10),
                                   (180, 300, 11)])
def test_volumes_around_the_lines(gpu, oracle_cpu, H, W, D):
    from cbmv_b200 import libmatchers as mtc
    o = oracle_cpu.mtc
    L, R = rand_pair(H + W + D, H, W, flat=True)
    sl, sr = o.sobel(L), o.sobel(R)
    for name, a, b, w in (("nccNister", L, R, 3), ("sadsob", sl, sr, 5), ("zsad", L, R, 5)):
        want = getattr(o, name)(a, b, D, w)
        for dtype in (np.float64, np.float32):
            dhw = getattr(mtc, name)(a, b, D, w, dtype=dtype, layout="DHW")
            hwd = getattr(mtc, name)(a, b, D, w, dtype=dtype, layout="HWD")
            assert np.array_equal(dhw, want.astype(dtype)), (name, dtype)
            assert np.array_equal(hwd, np.transpose(dhw, (1, 2, 0))), (name, dtype)
