"""The weight gradients' chains, split over a cluster between 8 and 64 tiles
of 128 samples: at the edges of that range and where four does not divide the
tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BLOCKS = [128 * 20, 128, 128 * 128, 128, 64 * 128, 64, 64, 1]


def _net_and_batch(act, tiles):
    from cbmv_b200.mlp import MlpParams, input_stats
    rng = np.random.default_rng(tiles)
    X = rng.normal(size=(128 * tiles, 20)).astype(np.float32) * np.linspace(0.5, 40, 20).astype(np.float32)
    y = ((X[:, 0] + 0.05 * X[:, 7] - 0.01 * X[:, 12]) > 0).astype(np.float32)
    net = MlpParams.init(1, *input_stats(X), act)
    net.views()["b1"][:] = 0.1
    return net, X, y


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("tiles", [7, 8, 9, 11, 63, 64, 65])
def test_gradients_around_the_split(gpu, act, tiles):
    """Each gradient block within 1e-3 of the float64 oracle that rounds to
    bf16 at the same points (the bound of the unsplit chains' tests), the same
    bits twice."""
    from cbmv_b200.mlp import MlpTrainer
    from oracle import mlp_ref
    net, X, y = _net_and_batch(act, tiles)
    tr = MlpTrainer(net, batch=len(X))
    Xt, yt = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    g, loss = tr.gradients(Xt, yt)
    again, _ = tr.gradients(Xt, yt)
    assert tr.status() == 0 and torch.equal(g, again)
    lref, gref, _ = mlp_ref.loss_and_grads(net.vec, X, y, act)
    assert abs(loss.item() - lref) < 1e-5 * max(1.0, abs(lref))
    got, o = g.cpu().numpy().astype(np.float64), 0
    for s in BLOCKS:
        a, b = got[o:o + s], gref[o:o + s]
        assert np.abs(a - b).max() / max(np.abs(b).max(), 1e-12) < 1e-3, (o, s)
        o += s


@pytest.mark.parametrize("tiles", [8, 16, 64])
def test_split_equals_the_mean_of_single_tiles(gpu, tiles):
    """A batch of 2^k tiles against the mean of its tiles' own gradients (the
    deltas differ by a power of two, so every operand has the same bits):
    float32 accumulation over at most 64 tiles, 512 additions of 2^-24 each
    against sums whose terms cancel tenfold at most: 3e-4."""
    from cbmv_b200.mlp import MlpTrainer
    net, X, y = _net_and_batch("gelu", tiles)
    Xt, yt = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    g = MlpTrainer(net, batch=len(X)).gradients(Xt, yt)[0].cpu().numpy().astype(np.float64)
    one = MlpTrainer(net, batch=128)
    parts = [one.gradients(Xt[i:i + 128].contiguous(), yt[i:i + 128].contiguous())[0].cpu().numpy().astype(np.float64)
             for i in range(0, len(X), 128)]
    want, o = np.mean(parts, axis=0), 0
    for s in BLOCKS:
        a, b = g[o:o + s], want[o:o + s]
        assert np.abs(a - b).max() <= 3e-4 * np.abs(b).max(), (o, s)
        o += s


@pytest.mark.parametrize("tiles", [2, 64])
def test_gradients_under_capture(gpu, tiles):
    """Both launches (the second set up beside the first) in a CUDA graph."""
    from cbmv_b200.mlp import MlpTrainer
    net, X, y = _net_and_batch("gelu", tiles)
    tr = MlpTrainer(net, batch=len(X))
    Xt, yt = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    want = tr.gradients(Xt, yt)[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, _ = tr.gradients(Xt, yt)
    for _ in range(2):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
