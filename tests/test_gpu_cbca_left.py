"""cbca on [D,H,W] where some of its tiles (32 columns, 16 rows, eight
disparities) have arms beyond the taps and others have not: the first are left
to a second launch, which finds them by a mark in the output.  The mark's bits
also stand in the input.  Against the oracle's sums in the reference's order:
equal."""
import numpy as np
import pytest

from test_gpu_cbca_any_arms import _dhw
from test_gpu_cbca_dhw import _arms

pytestmark = pytest.mark.gpu
MARK = np.array([0x7FA5C3E1], np.uint32).view(np.float32)[0]


@pytest.mark.parametrize("H,W,D", [(130, 200, 45), (97, 705, 13), (31, 33, 800)])
@pytest.mark.parametrize("direction", [-1, 1])
@pytest.mark.parametrize("part", ["rows", "columns", "pixel", "fraction"])
def test_tiles_left(gpu, oracle_cpu, H, W, D, part, direction):
    rng = np.random.default_rng(H + W)
    lc, rc = (_arms(rng, H, W, 6, 0) for _ in range(2))
    ll, lr = (_arms(rng, H, W, 25, 0) for _ in range(2))
    at = {"rows": np.s_[:, H // 2:], "columns": np.s_[:, :, :W // 3], "pixel": np.s_[:, H // 3, W // 2],
          "fraction": np.s_[:, H // 3, W // 2]}[part]
    if part == "fraction":
        lc[at] += np.float32(0.25)
    else:
        lc[at], rc[at] = ll[at], lr[at]
    v = rng.random((D, H, W)).astype(np.float32)
    v[:, :, ::32][rng.random(v[:, :, ::32].shape) < 0.01] = MARK
    with np.errstate(invalid="ignore"):
        _dhw(oracle_cpu, np.ascontiguousarray(lc), np.ascontiguousarray(rc), v, direction)
