"""cbca with arms that cbmv_cross does not give: arms that exclude their own
pixel, empty supports, arms longer than five pixels or than a byte counts.
Against the same float32 sums in numpy: equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F = np.float32


def _arms(rng, H, W, shift):
    """Intervals of 0 to 4 pixels that begin up to `shift` pixels beside their pixel, inside the image."""
    y, x = np.mgrid[0:H, 0:W]
    lo = np.clip(x + rng.integers(-shift, shift + 1, (H, W)), 0, W - 1)
    up = np.clip(y + rng.integers(-shift, shift + 1, (H, W)), 0, H - 1)
    return np.stack([lo - 1, np.minimum(lo + rng.integers(0, 5, (H, W)), W), up - 1,
                     np.minimum(up + rng.integers(0, 5, (H, W)), H)]).astype(np.float32)


def _separable(lc, rc, v, direction):
    """Row sums over the taps -5..5 of each support row, then column sums over
    those of the support column, divided by the rows' pixels."""
    H, W, D = v.shape
    out = v.copy()
    taps = range(-5, 6)

    def row(y, x, d):
        s, xm = d * direction, x + d * direction
        return int(max(lc[0, y, x], rc[0, y, xm] - s)), int(min(lc[1, y, x], rc[1, y, xm] - s))

    for d in range(D):
        for x in range(W):
            if not 0 <= x + d * direction < W:
                continue
            sums = np.zeros(H, F)
            for y in range(H):
                lo, hi = row(y, x, d)
                for k in taps:
                    if lo < x + k < hi:
                        sums[y] += v[y, x + k, d]
            for y in range(H):
                lo = int(max(lc[2, y, x], rc[2, y, x + d * direction]))
                hi = int(min(lc[3, y, x], rc[3, y, x + d * direction]))
                s, n = F(0), 0
                for k in taps:
                    if lo < y + k < hi:
                        s += sums[y + k]
                        a, b = row(y + k, x, d)
                        n += max(b - a - 1, 0)
                out[y, x, d] = s / F(n)
    return out


def _dhw(oracle_cpu, lc, rc, v, direction):
    """cbmv_cbca on [D,H,W] and the reference-order sums of the oracle."""
    from cbmv_b200 import _lib
    D, H, W = v.shape
    want, v64 = np.empty(v.shape), v.astype(np.float64)
    oracle_cpu.lib().orc_cbca(lc.ctypes.data, rc.ctypes.data, v64.ctypes.data, D, H, W, direction, want.ctypes.data)
    tl, tr, tv = (torch.from_numpy(a).cuda() for a in (lc, rc, v))
    got = torch.empty_like(tv)
    _lib.call("cbmv_cbca", tl.data_ptr(), tr.data_ptr(), tv.data_ptr(), H, W, D, _lib.DHW, direction, got.data_ptr(),
              None)
    assert np.array_equal(got.cpu().numpy(), want.astype(F), equal_nan=True)


@pytest.mark.parametrize("direction", [-1, 1])
@pytest.mark.parametrize("H,W,D,shift", [(9, 17, 5, 2), (150, 97, 57, 2), (14, 430, 140, 200), (310, 27, 100, 150)])
def test_dhw_with_any_arms(gpu, oracle_cpu, H, W, D, shift, direction):
    """The supports of a shift of 150 pixels and more lie beyond the byte that
    holds a relative arm."""
    rng = np.random.default_rng(H + W)
    y, x = np.mgrid[0:H, 0:W]
    lo = np.clip(x + shift + rng.integers(-2, 3, (H, W)), 0, W - 1)
    up = np.clip(y - shift + rng.integers(-2, 3, (H, W)), 0, H - 1)
    lc, rc = (np.stack([lo - 1, np.minimum(lo + rng.integers(2, 7, (H, W)), W), up - 1,
                        np.minimum(up + rng.integers(2, 7, (H, W)), H)]).astype(F) for _ in range(2))
    _dhw(oracle_cpu, lc, rc, rng.random((D, H, W)).astype(F), direction)


# beyond 800,000 values the sums run in tiles of 32 columns, 16 rows and eight disparities
@pytest.mark.parametrize("H,W,D,reach,fraction", [(113, 97, 73, 6, 0), (112, 96, 80, 6, 0), (127, 129, 49, 9, 0),
                                                  (66, 130, 97, 6, 0.25), (700, 701, 3, 6, 0), (710, 705, 2, 6, 0)])
@pytest.mark.parametrize("direction", [-1, 1])
def test_dhw_at_tile_edges(gpu, oracle_cpu, H, W, D, reach, fraction, direction):
    from test_gpu_cbca_dhw import _arms as arms
    rng = np.random.default_rng(H * W + D)
    lc, rc = (np.ascontiguousarray(arms(rng, H, W, reach, fraction)) for _ in range(2))
    v = rng.random((D, H, W)).astype(F)
    v[rng.random(v.shape) < 0.002] = np.inf
    _dhw(oracle_cpu, lc, rc, v, direction)


@pytest.mark.parametrize("direction", [-1, 1])
@pytest.mark.parametrize("H,W,D,shift", [(9, 17, 5, 1), (14, 35, 3, 3), (11, 40, 2, 9)])
def test_separable_with_any_arms(gpu, H, W, D, shift, direction):
    from cbmv_b200 import _lib
    rng = np.random.default_rng(H * W + shift)
    lc, rc = _arms(rng, H, W, shift), _arms(rng, H, W, shift)
    v = rng.random((H, W, D)).astype(np.float32)
    with np.errstate(all="ignore"):
        want = _separable(lc, rc, v, direction)
    tl, tr, tv = (torch.from_numpy(a).cuda() for a in (lc, rc, v))
    got = torch.empty_like(tv)
    _lib.call("cbmv_cbca_separable", tl.data_ptr(), tr.data_ptr(), tv.data_ptr(), H, W, D, 6, direction, got.data_ptr(),
              None)
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)
