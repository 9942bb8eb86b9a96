"""A caller's cost volume is read where it lies when it is 16-byte aligned
and copied when it is not: the same disparity either way, for every number of
passes after it, and the volume is left as it was."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

H, W, D = 20, 45, 24


def _at(v, off):
    buf = torch.empty(v.numel() + 4, device="cuda")
    out = buf[off:off + v.numel()].view(v.shape)
    out.copy_(v)
    return out


@pytest.mark.parametrize("passes", [(0, 0, 0), (0, 1, 0), (1, 0, 0), (0, 1, 1), (1, 1, 1), (0, 2, 4)])
@pytest.mark.parametrize("interpolate", [0, 1])
def test_run_post(gpu, passes, interpolate):
    from cbmv_b200 import _lib
    from cbmv_b200.pipeline import StereoPipeline
    rng = np.random.default_rng(1)
    l, r = (torch.from_numpy(rng.integers(90, 110, (H, W)).astype(np.uint8)).cuda() for _ in range(2))
    cost = torch.from_numpy(rng.random((H, W, D)).astype(np.float32)).cuda()
    prm = _lib.default_params(cbca_i1=passes[0], sgm_i=passes[1], cbca_i2=passes[2], interpolate=interpolate)
    pipe, got = StereoPipeline(params=prm), []
    for off in (0, 1, 2):
        c = _at(cost, off)
        got.append(pipe.run_post(l, r, c))
        assert torch.equal(c, cost)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("interpolate", [0, 1])
def test_probability_volume(gpu, small_pair, interpolate):
    import os
    from cbmv_b200 import _lib
    from cbmv_b200.mlp import GpuMlp
    from cbmv_b200.pipeline import StereoPipeline
    net = GpuMlp.load(os.path.join(os.path.dirname(__file__), "golden", "mlp_gelu_694x554.npz"))
    L, R = (torch.from_numpy(v).cuda() for v in small_pair[:2])
    h, w = L.shape
    pipe = StereoPipeline(params=_lib.default_params(interpolate=interpolate))
    want = pipe.run_mlp(net, L, R, D)
    probs = []
    for off in (0, 1):
        prob = _at(torch.zeros(h, w, D, device="cuda"), off)
        assert torch.equal(pipe.run_mlp(net, L, R, D, prob_out=prob), want)
        probs.append(prob)
    assert torch.equal(probs[0], probs[1])
    assert torch.equal(pipe.run_post(L, R, probs[0]), want)
