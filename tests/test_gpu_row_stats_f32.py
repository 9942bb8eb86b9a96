"""The learned path's row statistics over every number of registers per lane
(vectors of four where D is a multiple of four) and pixel counts that leave a
warp's last pixels empty: ratio and likelihood of both views from the float32
volumes themselves in float64, to 1e-5 relative above 1e-11 (the bar of the
learned features' own test: the float32 argument and the approximate
exponential stay within it)."""
import numpy as np
import pytest
import torch

from conftest import rand_pair

pytestmark = pytest.mark.gpu

EPS, SIGMA = (0.01, 1.01, 0.01, 0.01), (128.0, 0.02, 20000.0, 20000.0)


@pytest.mark.parametrize("H,W,D", [(13, 15, 1), (12, 33, 31), (13, 37, 33), (13, 41, 70), (13, 301, 97), (12, 31, 130),
                                   (13, 35, 161), (12, 33, 222), (13, 31, 255), (13, 31, 132), (12, 33, 256),
                                   (13, 31, 260), (12, 33, 388), (13, 31, 512), (13, 33, 301), (12, 21, 516)])
def test_statistics_of_both_views(gpu, H, W, D):
    from cbmv_b200.pipeline import StereoPipeline
    L, R = rand_pair(D, H, W)
    pipe = StereoPipeline()
    vols = pipe.volumes_f32(L, R, D).cpu().numpy().astype(np.float64)
    got = pipe.features_at(L, R, D, np.arange(H * W * D, dtype=np.int64), learned=True).cpu().numpy().astype(np.float64)
    got = got.reshape(H, W, D, 20)
    x, d = np.arange(W)[:, None], np.arange(D)
    inside = (x >= d)[None]
    back = np.broadcast_to(np.maximum(x - d, 0)[None], (H, W, D))
    for m in range(4):
        c = vols[m]
        right = np.full_like(c, c[0, 0, 0])
        for k in range(min(D, W)):
            right[:, :W - k, k] = c[:, k:, k]
        for view, v in enumerate((c, right)):
            mn = v.min(2, keepdims=True)
            e = np.exp(-((v - mn) ** 2) / SIGMA[m])
            none = mn == 2147483648.0
            want = [np.where(none, 0, (mn + EPS[m]) / (v + EPS[m])), np.where(none, 0, e / e.sum(2, keepdims=True))]
            if view:
                want = [np.where(inside, np.take_along_axis(w, back, axis=1), 0) for w in want]
            for w, col in zip(want, (4 + m, 8 + m) if view == 0 else (12 + m, 16 + m)):
                err = np.abs(got[..., col] - w)
                assert (err <= 1e-5 * np.abs(w) + 1e-11).all(), (m, view, col, err.max())
