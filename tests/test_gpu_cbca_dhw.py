"""cbca on [D,H,W] volumes at the edges of its tiles (32 columns, 16 rows,
eight disparities), with arms inside and beyond its five taps, costs that are
infinite outside a support, and arms that are no whole numbers, against the
same sums in numpy.  The sums are float32 in one order: equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _arms(rng, H, W, reach, fraction):
    y, x = np.mgrid[0:H, 0:W]
    a = np.stack([np.maximum(x - rng.integers(1, reach + 1, (H, W)), -1), np.minimum(x + rng.integers(1, reach + 1, (H, W)), W),
                  np.maximum(y - rng.integers(1, reach + 1, (H, W)), -1),
                  np.minimum(y + rng.integers(1, reach + 1, (H, W)), H)]).astype(np.float32)
    return a + np.float32(fraction) * (rng.random(a.shape) < 0.01)


def _reference(lc, rc, v, direction):
    D, H, W = v.shape
    out = v.copy()
    f = np.float32
    for d in range(D):
        for y in range(H):
            for x in range(W):
                xm = x + d * direction
                if not 0 <= xm < W:
                    continue
                s, n = f(0), 0
                for yy in range(int(max(lc[2, y, x], rc[2, y, xm])) + 1, int(min(lc[3, y, x], rc[3, y, xm]))):
                    lo = int(max(lc[0, yy, x], rc[0, yy, xm] - f(d * direction))) + 1
                    hi = int(min(lc[1, yy, x], rc[1, yy, xm] - f(d * direction)))
                    for xx in range(lo, hi):
                        s += v[d, yy, xx]
                        n += 1
                out[d, y, x] = s / f(n)
    return out


@pytest.mark.parametrize("H,W,D,reach,fraction", [(1, 1, 1, 6, 0), (17, 33, 9, 6, 0), (16, 32, 8, 6, 0), (31, 40, 7, 9, 0),
                                                  (18, 34, 3, 6, 0.25)])
@pytest.mark.parametrize("direction", [-1, 1])
def test_cbca_dhw(gpu, H, W, D, reach, fraction, direction):
    from cbmv_b200 import _lib
    rng = np.random.default_rng(H * W + D)
    lc, rc = _arms(rng, H, W, reach, fraction), _arms(rng, H, W, reach, fraction)
    v = rng.random((D, H, W)).astype(np.float32)
    v[rng.random(v.shape) < 0.002] = np.inf
    with np.errstate(all="ignore"):
        want = _reference(lc, rc, v, direction)
    tl, tr, tv = (torch.from_numpy(a).cuda() for a in (lc, rc, v))
    got = torch.empty_like(tv)
    _lib.call("cbmv_cbca", tl.data_ptr(), tr.data_ptr(), tv.data_ptr(), H, W, D, _lib.DHW, direction, got.data_ptr(),
              None)
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)
