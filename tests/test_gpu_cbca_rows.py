"""Rows per CBCA tile: an upper bound, so that a batch tuned with an explicit
bound keeps the short tiles of small pairs; and the passes with 32, 16 and 8
rows at odd sizes, the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(H, W, D, rows):
    from cbmv_b200 import _lib
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(H + D)
    l, r = (torch.from_numpy(rng.integers(90, 96, (H, W)).astype(np.uint8)).cuda() for _ in range(2))
    cost = torch.from_numpy(rng.random((H, W, D)).astype(np.float32)).cuda()
    pipe = StereoPipeline(params=_lib.default_params(cbca_rows=rows))
    return lambda: pipe.run_post(l, r, cost)


def _passes(call):
    """Names of the CBCA passes' kernels of one call."""
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = {e.key for e in prof.key_averages() if "cbca_hwd_mask_kernel" in e.key}
    if not names:
        pytest.skip("the profiler lists no kernels here")
    return names


# 32-row tiles fill the GPU from 296 on
@pytest.mark.parametrize("H,W,D,taken", [(64, 96, 16, {0: 8, 16: 8, 32: 8}), (95, 203, 64, {0: 16, 16: 16, 32: 16}),
                                         (131, 203, 100, {0: 32, 16: 16, 32: 32})])
def test_rows_are_an_upper_bound(gpu, H, W, D, taken):
    for rows, want in taken.items():
        names = _passes(_run(H, W, D, rows))
        assert all("cbca_hwd_mask_kernel<%d>" % want in n for n in names), (rows, names)


@pytest.mark.parametrize("H,W,D", [(95, 203, 64), (131, 203, 100), (129, 205, 97)])
def test_rows_do_not_change_the_result(gpu, H, W, D):
    got = [_run(H, W, D, rows)().cpu() for rows in (0, 16, 32)]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("H,W,D", [(95, 203, 64), (131, 203, 100)])
def test_long_tiles_equal_the_model(gpu, H, W, D):
    from cbmv_b200 import _lib
    from oracle import post_model
    from test_gpu_cbca_masked import _arms
    rng = np.random.default_rng(D)
    lc, rc = _arms(rng, H, W), _arms(rng, H, W)
    v = torch.from_numpy(rng.random((H, W, D)).astype(np.float32)).cuda()
    out = torch.empty_like(v)
    _lib.call("cbmv_cbca_separable", lc.data_ptr(), rc.data_ptr(), v.data_ptr(), H, W, D, 6, -1, out.data_ptr(), None)
    want = post_model.cbca_separable(lc.cpu().numpy(), rc.cpu().numpy(), v.cpu().numpy(), -1, 5)
    assert np.array_equal(out.cpu().numpy(), want)
