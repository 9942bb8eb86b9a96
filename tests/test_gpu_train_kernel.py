"""The fused training kernel at the edges of its tiling: one 128-sample
tile, and more tiles than SMs (a CTA accumulates two), on samples that
start 4 bytes off a 16-byte boundary."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _toy(seed, n):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, 20)).astype(np.float32) * np.linspace(0.5, 40, 20).astype(np.float32)
    X[rng.random((n, 20)) < 0.02] = 2147483648.0  # cost sentinels
    y = ((X[:, 0] + 0.05 * X[:, 7] - 0.01 * X[:, 12]) > 0).astype(np.float32)
    return X, y


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("extra_tiles", [None, 1])
def test_gradients_and_step_at_tile_edges(gpu, act, extra_tiles):
    """Every gradient block within 1e-3 of the float64 oracle that rounds to
    bf16 at the same points (the bound of the 256-sample test: float32
    accumulation moves a bf16 rounding here and there), the same bits twice,
    and a step that applies Adam's first update to exactly these gradients."""
    from cbmv_b200.mlp import MlpParams, MlpTrainer, input_stats
    from oracle import mlp_ref
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 128 if extra_tiles is None else 128 * (sms + extra_tiles)
    X, y = _toy(3, n)
    cap, mu, sd = input_stats(X)
    net = MlpParams.init(1, cap, mu, sd, act)
    v = net.views()
    v["b1"][:] = 0.1
    v["b2"][:] = -0.05
    v["b3"][:] = 0.02
    v["b4"][:] = 0.3
    buf = torch.empty(n * 20 + 1, device="cuda")
    Xt = buf[1:].view(n, 20)
    Xt.copy_(torch.from_numpy(X))
    yt = torch.from_numpy(y).cuda()
    tr = MlpTrainer(net, batch=n)
    g, loss = tr.gradients(Xt, yt)
    again, _ = tr.gradients(Xt, yt)
    assert tr.status() == 0
    assert torch.equal(g, again)
    lref, gref, _ = mlp_ref.loss_and_grads(net.vec, X, y, act)
    assert abs(loss.item() - lref) < 1e-5 * max(1.0, abs(lref))
    got, o = g.cpu().numpy().astype(np.float64), 0
    for s in [128 * 20, 128, 128 * 128, 128, 64 * 128, 64, 64, 1]:
        a, b = got[o:o + s], gref[o:o + s]
        assert np.abs(a - b).max() / max(np.abs(b).max(), 1e-12) < 1e-3, (o, s)
        o += s
    # Adam's first step moves every parameter by lr * g / (|g| + eps')
    lr = 1e-3
    assert tr.step(Xt, yt, lr).item() == loss.item()
    moved = (tr.params().vec - net.vec)[60:].astype(np.float64)
    want = -lr * got / (np.abs(got) + 1e-8)
    # float32 rounding of the parameters (|p| < 1) and of the bias corrections
    assert np.abs(moved - want).max() < 1e-6
