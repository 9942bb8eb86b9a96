"""Where a caller's cost volume lies: in pageable host memory it is an error
before any launch, in pinned host memory it is copied as any volume that the
passes cannot use in place."""
import ctypes

import pytest
import torch

from conftest import rand_pair

pytestmark = pytest.mark.gpu
H, W, D = 40, 52, 16


def test_volumes_in_host_memory(gpu):
    import os
    from cbmv_b200 import _lib
    from cbmv_b200.mlp import GpuMlp
    from cbmv_b200.pipeline import StereoPipeline
    from conftest import GOLDEN
    net = GpuMlp.load(os.path.join(GOLDEN, "mlp_gelu_694x554.npz"))
    L, R = (torch.from_numpy(a).cuda() for a in rand_pair(4, H, W, flat=True))
    pipe = StereoPipeline()
    prob = torch.empty(H, W, D, device="cuda")
    want = pipe.run_mlp(net, L, R, D, prob_out=prob).clone()
    pageable, pinned = torch.empty(H, W, D), torch.empty(H, W, D).pin_memory()
    disp = torch.empty(H, W, device="cuda")

    def post(cost):
        _lib.call("cbmv_run_post", pipe.ctx, ctypes.byref(pipe.params), L.data_ptr(), R.data_ptr(), H, W, D,
                  cost.data_ptr(), disp.data_ptr())

    for call in (lambda: pipe.run_mlp(net, L, R, D, prob_out=pageable), lambda: post(pageable)):
        pageable.copy_(prob)
        try:
            call()  # a device that reads pageable memory takes it
            torch.cuda.synchronize()
        except _lib.CbmvError as e:
            assert "pageable" in str(e)
        else:
            assert torch.equal(pageable, prob.cpu())
    assert torch.equal(pipe.run_mlp(net, L, R, D, prob_out=pinned), want)
    torch.cuda.synchronize()
    assert torch.equal(pinned, prob.cpu())
    post(pinned)
    assert torch.equal(disp, want)
    post(prob)
    assert torch.equal(disp, want)
