"""The float64 features around the edges of the row-statistics kernels
(32 right pixels per warp, 4 / 8 / any number of 32-disparity registers) on
volumes with what a caller's own may hold: infinities, huge and tiny costs,
sentinel rows.  Against the formulas in numpy: the float32 rounding of a
float64 chain that may differ from numpy's by a few float64 units, so at most
one float32 unit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RAND_MAX = 2147483647.0
EPS, SIGMA = (0.01, 1.01, 0.01, 0.01), (128.0, 0.02, 20000.0, 20000.0)


def _reference(vols):
    H, W, D = vols[0].shape
    out = np.zeros((H, W, D, 20))
    x, d = np.arange(W)[:, None], np.arange(D)
    with np.errstate(all="ignore"):
        for m, c in enumerate(vols):
            right = np.full_like(c, c[0, 0, 0])
            for k in range(min(D, W)):
                right[:, :W - k, k] = c[:, k:, k]

            def conf(v, row):
                mn = np.minimum(np.fmin.reduce(row, axis=2), RAND_MAX)[:, :, None]
                den = np.exp(-((row - mn) ** 2) / SIGMA[m]).sum(2)[:, :, None]
                r = np.where(mn == RAND_MAX, 0, (mn + EPS[m]) / (v + EPS[m]))
                return r, np.where(mn == RAND_MAX, 0, np.exp(-((v - mn) ** 2) / SIGMA[m]) / den)

            out[..., m] = c
            out[..., 4 + m], out[..., 8 + m] = conf(c, c)
            r, l = conf(right, right)
            back = np.broadcast_to(np.maximum(x - d, 0)[None], c.shape)
            for j, v in ((12 + m, r), (16 + m, l)):
                out[..., j] = np.where(x >= d, np.take_along_axis(v, back, axis=1), 0)
        return out.reshape(-1, 20).astype(np.float32)


@pytest.mark.parametrize("H,W,D", [(3, 33, 1), (2, 31, 33), (3, 64, 128), (2, 70, 130), (1, 40, 260)])
def test_features_of_any_volume(gpu, H, W, D):
    from cbmv_b200 import libfeatextract as fte
    rng = np.random.default_rng(H * W * D)
    vols = []
    for m in range(4):
        v = rng.random((H, W, D)) * (120, 2, 3000, 900)[m]
        v[rng.random(v.shape) < 0.1] = RAND_MAX
        v[rng.random(v.shape) < 0.03] = np.inf
        v[rng.random(v.shape) < 0.03] = 1e200
        v[rng.random(v.shape) < 0.03] *= 1e-150
        v[rng.random((H, W)) < 0.1] = RAND_MAX
        vols.append(v)
    got, want = fte.features(*vols), _reference(vols)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    a, b = got[ok], want[ok]
    assert np.array_equal(np.isinf(a), np.isinf(b))
    fin = np.isfinite(b)
    assert np.abs(a[fin].view(np.int32).astype(np.int64) - b[fin].view(np.int32).astype(np.int64)).max() <= 1
