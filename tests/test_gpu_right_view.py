"""The right view's cost of the left-right check at the edges of its tiles (64
pixels, 32 disparities) and the winner-take-all over vector and single loads:
ties take the first disparity, +inf and NaN are never a minimum."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 3, 4, 31, 32, 36, 128, 130, 132, 260])
@pytest.mark.parametrize("off", [0, 1])
def test_winner_take_all(gpu, D, off):
    from cbmv_b200 import _lib
    rng = np.random.default_rng(D)
    H, W = 5, 77
    v = rng.integers(0, 4 + D // 8, (H, W, D)).astype(np.float32)
    v[0] = np.inf
    v[1][rng.random((W, D)) < 0.5] = np.nan
    v[2] = np.nan
    v[3][:, : D // 2] = 0.0
    v[3][rng.random((W, D)) < 0.3] = -0.0
    buf = torch.empty(v.size + 4, device="cuda")
    c = buf[off:off + v.size].view(v.shape)
    c.copy_(torch.from_numpy(v))
    out = torch.empty((H, W), device="cuda")
    _lib.call("cbmv_wta", c.data_ptr(), H, W, D, _lib.HWD, out.data_ptr(), None)
    want = np.argmin(np.where(np.isnan(v), np.inf, v), 2)
    assert np.array_equal(out.cpu().numpy(), want.astype(np.float32))


@pytest.mark.parametrize("W,D", [(12, 5), (63, 31), (64, 32), (65, 33), (128, 70), (130, 40), (40, 64)])
def test_left_right_check_of_the_two_views(gpu, W, D):
    """With no passes on the costs the _interp chain is the two views'
    argmins, the check and the fills."""
    from cbmv_b200 import _lib
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(W)
    H = 13
    cost = rng.random((H, W, D)).astype(np.float32)
    img = rng.integers(0, 256, (2, H, W)).astype(np.uint8)
    prm = _lib.default_params(interpolate=1, sgm_i=0, cbca_i1=0, cbca_i2=0, median_i=0, blur_t=1e-6)
    got = StereoPipeline(params=prm).run_post(img[0], img[1], cost)
    right = np.full_like(cost, cost[0, 0, 0])
    for d in range(D):
        right[:, : max(W - d, 0), d] = cost[:, d:, d]
    d0, d1 = (torch.from_numpy(np.argmin(v, 2).astype(np.float32)).cuda() for v in (cost, right))
    o, a, b = (torch.empty((H, W), device="cuda") for _ in range(3))
    _lib.call("cbmv_outlier_detection", d0.data_ptr(), d1.data_ptr(), H, W, D, o.data_ptr(), None)
    _lib.call("cbmv_interpolate_mismatch", d0.data_ptr(), o.data_ptr(), H, W, a.data_ptr(), None)
    _lib.call("cbmv_interpolate_occlusion", a.data_ptr(), o.data_ptr(), H, W, b.data_ptr(), None)
    # the blur averages equal values only: at most its rounding
    assert np.abs(got - b.cpu().numpy()).max() < 1e-3
