"""The terms of both images formed in one launch, and the CBCA's tile rows,
at sizes around their tiles (32 x 16 pixels; 8, 16 or 32 rows) and from images
that start at any byte: the volumes equal the general windows' route and the
oracle, the post-processing equals the single operations in the same order."""
import numpy as np
import pytest
import torch

from conftest import rand_pair

pytestmark = pytest.mark.gpu


def _at(img, off):
    """The image on the device, its first byte `off` past an aligned one."""
    buf = torch.empty(img.size + 16, dtype=torch.uint8, device="cuda")
    view = buf[off:off + img.size].view(img.shape)
    view.copy_(torch.from_numpy(img))
    return view


@pytest.mark.parametrize("H,W,off", [(12, 15, 1), (13, 40, 2), (12, 12, 3), (16, 32, 0), (17, 33, 1),
                                     (33, 64, 5), (50, 95, 7)])
def test_volumes_around_tiles(gpu, oracle_cpu, H, W, off):
    from cbmv_b200.pipeline import StereoPipeline
    o, D = oracle_cpu.mtc, 9
    L, R = rand_pair(H * W, H, W)
    got = StereoPipeline().volumes_f32(_at(L, off), _at(R, (off + 1) % 8), D).cpu().numpy()
    sl, sr = o.sobel(L), o.sobel(R)
    want = [o.census(L, R, D, 11), np.transpose(o.nccNister(L, R, D, 3), (1, 2, 0)),
            np.transpose(o.sadsob(sl, sr, D, 5), (1, 2, 0))]
    for k in range(3):
        assert np.array_equal(got[k], want[k].astype(np.float32)), k


@pytest.mark.parametrize("H,W,D,off", [(12, 12, 2, 0), (12, 13, 5, 1), (16, 31, 33, 2), (17, 32, 32, 3), (33, 40, 40, 5)])
def test_post_equals_single_operations(gpu, H, W, D, off):
    from cbmv_b200 import _lib
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(H * W)
    imgs = [(rng.integers(0, 3, (H, W)) * 90 + rng.integers(0, 5, (H, W))).astype(np.uint8) for _ in range(2)]
    cost = torch.from_numpy(rng.random((H, W, D)).astype(np.float32)).cuda()
    prm = dict(exact_cbca=1, sgm_i=0, cbca_i1=1, cbca_i2=0, median_i=0, blur_t=1e-6)
    l, r = _at(imgs[0], off), _at(imgs[1], (off + 3) % 8)
    got = StereoPipeline(params=_lib.default_params(**prm)).run_post(l, r, cost)
    p = _lib.default_params(**prm)
    arms = []
    for im in imgs:
        # the float32 mean and standard deviation of the exact integer sums
        n, s, q = im.size, int(im.astype(np.int64).sum()), int((im.astype(np.int64) ** 2).sum())
        m = np.float64(s) / n
        sd = np.sqrt(max(np.float64(q) / n - m * m, 0.0))
        with np.errstate(divide="ignore", invalid="ignore"):
            x = (im.astype(np.float32) - np.float32(m)) / np.float32(sd)
        a = torch.empty((4, H, W), device="cuda")
        _lib.call("cbmv_cross", torch.from_numpy(x).cuda().data_ptr(), H, W, p.L1, p.tau1, a.data_ptr(), None)
        arms.append(a)
    out = torch.empty_like(cost)
    _lib.call("cbmv_cbca", arms[0].data_ptr(), arms[1].data_ptr(), cost.data_ptr(), H, W, D, _lib.HWD, -1,
              out.data_ptr(), None)
    want = np.argmin(out.cpu().numpy(), 2)
    # a blur threshold this small averages equal values only: the subpixel disparity, half a step from the minimum at most
    assert np.abs(got.cpu().numpy() - want).max() <= 0.501


@pytest.mark.parametrize("H,W,D", [(12, 16, 32), (15, 13, 5), (16, 31, 33), (17, 17, 40), (33, 40, 40), (70, 64, 64)])
def test_tile_rows_do_not_change_the_result(gpu, H, W, D):
    from cbmv_b200 import _lib
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(D)
    l, r = (torch.from_numpy(rng.integers(90, 96, (H, W)).astype(np.uint8)).cuda() for _ in range(2))
    cost = torch.from_numpy(rng.random((H, W, D)).astype(np.float32)).cuda()
    got = [StereoPipeline(params=_lib.default_params(cbca_rows=k)).run_post(l, r, cost).cpu().numpy() for k in (0, 16, 32)]
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
