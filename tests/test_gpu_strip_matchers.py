"""The strip matchers at the edges of their strips (32 or 16 columns) and
disparity blocks (32), in both layouts and output types, against the oracle:
float64 equal, float32 the rounding of the float64 value (ZSAD of the
learned path: the exact quotient, at most one unit from it)."""
import numpy as np
import pytest

from conftest import rand_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,D", [(12, 31, 1), (13, 32, 31), (17, 33, 33), (16, 65, 32), (14, 97, 70), (5, 40, 8),
                                   (30, 10, 12)])
def test_volumes_at_strip_edges(gpu, oracle_cpu, H, W, D):
    from cbmv_b200 import libmatchers as mtc
    o = oracle_cpu.mtc
    L, R = rand_pair(H * W + D, H, W, flat=H > 12 and W > 12)
    sl, sr = o.sobel(L), o.sobel(R)
    want = [o.census(L, R, D, 11), np.transpose(o.nccNister(L, R, D, 3), (1, 2, 0)),
            np.transpose(o.sadsob(sl, sr, D, 5), (1, 2, 0)), np.transpose(o.zsad(L, R, D, 5), (1, 2, 0))]
    for k, (fn, a, b, w) in enumerate([(mtc.census, L, R, 11), (mtc.nccNister, L, R, 3), (mtc.sadsob, sl, sr, 5),
                                       (mtc.zsad, L, R, 5)]):
        for dtype in (np.float64, np.float32):
            hwd = fn(a, b, D, w, dtype=dtype, layout="HWD")
            assert np.array_equal(hwd, want[k].astype(dtype)), (k, dtype)
            dhw = fn(a, b, D, w, dtype=dtype, layout="DHW")
            assert np.array_equal(dhw, np.transpose(hwd, (2, 0, 1))), (k, dtype)


def test_sadsob_beyond_image_gradients(gpu, oracle_cpu):
    """Integer responses outside the range of a Sobel filter of 8-bit pixels."""
    from cbmv_b200 import libmatchers as mtc
    rng = np.random.default_rng(3)
    sl, sr = (rng.integers(-2 ** 25, 2 ** 25, (20, 50)).astype(np.float64) for _ in range(2))
    assert np.array_equal(mtc.sadsob(sl, sr, 40, 5), oracle_cpu.mtc.sadsob(sl, sr, 40, 5))


@pytest.mark.parametrize("H,W,D", [(13, 33, 31), (40, 100, 70)])
def test_learned_zsad_of_extreme_windows(gpu, oracle_cpu, H, W, D):
    """Black and white pixels: the largest window sums of either sign."""
    from cbmv_b200 import libmatchers as mtc
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(H)
    L, R = (np.where(rng.random((H, W)) < p, 0, 255).astype(np.uint8) for p in (0.1, 0.9))
    got = StereoPipeline().volumes_f32(L, R, D).cpu().numpy()[3]
    want = np.transpose(oracle_cpu.mtc.zsad(L, R, D, 5), (1, 2, 0)).astype(np.float32)
    assert np.abs(got.view(np.int32).astype(np.int64) - want.view(np.int32).astype(np.int64)).max() <= 1


@pytest.mark.parametrize("D,H,W", [(1, 40, 33), (70, 5, 31), (33, 64, 32)])
def test_swap_axes_at_tile_edges(gpu, D, H, W):
    from cbmv_b200 import libfeatextract as fte
    v = np.random.default_rng(1).random((D, H, W))
    assert np.array_equal(fte.swap_axes(v), np.transpose(v, (1, 2, 0)))
    assert np.array_equal(fte.swap_axes_back(np.transpose(v, (1, 2, 0))), v)
