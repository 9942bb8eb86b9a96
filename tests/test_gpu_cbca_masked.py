"""The CBCA pass from precomputed supports at the edges of its tiles, on
values whose quotients the short division rounds as the division does, and on
values where it does not (zeros, subnormals, the largest floats, infinities,
NaN): the same bits as the float32 model of its summation order."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _arms(rng, H, W):
    img = (np.kron(rng.integers(0, 3, (H // 3 + 1, W // 4 + 1)), np.ones((3, 4)))[:H, :W]
           + rng.random((H, W)) * 0.08).astype(np.float32)
    from cbmv_b200 import _lib
    t, a = torch.from_numpy(img).cuda(), torch.empty(4, H, W, device="cuda")
    _lib.call("cbmv_cross", t.data_ptr(), H, W, 6, 0.07, a.data_ptr(), None)
    return a


@pytest.mark.parametrize("kind", ["plain", "wide", "special"])
@pytest.mark.parametrize("H,W,D", [(1, 5, 33), (7, 8, 32), (9, 17, 31), (33, 21, 40), (32, 26, 64), (70, 130, 70)])
@pytest.mark.parametrize("direction", [-1, 1])
def test_masked_pass_equals_model(gpu, H, W, D, kind, direction):
    from cbmv_b200 import _lib
    from oracle import post_model
    rng = np.random.default_rng(H * W + D)
    lc, rc = _arms(rng, H, W), _arms(rng, H, W)
    vol = rng.random((H, W, D)).astype(np.float32)
    if kind == "wide":
        vol *= np.exp2(rng.integers(-148, 120, vol.shape)).astype(np.float32)
    elif kind == "special":
        special = np.array([0, -0.0, 1e-45, -1e-40, 3e38, -3e38, np.inf, -np.inf, np.nan], np.float32)
        at = rng.random(vol.shape) < 0.02
        vol[at] = rng.choice(special, at.sum())
    v = torch.from_numpy(vol).cuda()
    out = torch.empty_like(v)
    _lib.call("cbmv_cbca_separable", lc.data_ptr(), rc.data_ptr(), v.data_ptr(), H, W, D, 6, direction,
              out.data_ptr(), None)
    with np.errstate(all="ignore"):
        want = post_model.cbca_separable(lc.cpu().numpy(), rc.cpu().numpy(), vol, direction, 5)
    got = out.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.int32), want[ok].view(np.int32))
