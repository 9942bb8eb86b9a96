"""The forest's device layout: trees with more groups than an entry can
number (subtrees reached by jumps), and the fused classifier at the edges of
its tiles, against the flat forest's own walk.  Leaves are indices and
probabilities sums of the same float64 values in the same order: equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_tree_beyond_one_segment(gpu):
    """A complete tree of depth 20 (349,525 blocks, 1,048,576 leaves) beside a
    single-leaf tree."""
    from cbmv_b200.forest import FlatForest
    from cbmv_b200.forest_gpu import GpuForest
    rng = np.random.default_rng(5)
    depth, F = 20, 20
    inner = 2 ** depth - 1
    n = 2 ** (depth + 1) - 1
    i = np.arange(n)
    level = np.floor(np.log2(i + 1)).astype(int)
    feature = np.where(i < inner, level % F, -2)
    threshold = np.where(i < inner, rng.normal(size=n), -2.0)
    left, right = np.where(i < inner, 2 * i + 1, -1), np.where(i < inner, 2 * i + 2, -1)
    value = rng.random(n)
    ff = FlatForest(np.array([0, n]), np.append(feature, -2), np.append(threshold, -2.0), np.append(left, -1),
                    np.append(right, -1), np.append(value, 0.25), n_features=F)
    X = rng.normal(size=(3001, F)).astype(np.float32)
    at = np.zeros(len(X), np.int64)
    for _ in range(depth):
        at = np.where(X[np.arange(len(X)), feature[at]].astype(np.float64) <= threshold[at], left[at], right[at])
    gf = GpuForest(ff)
    assert np.array_equal(gf.apply(X), np.stack([at, np.zeros_like(at)], 1))
    assert np.array_equal(gf.predict_proba(X)[:, 0], (value[at] + 0.25) / 2)
    assert np.array_equal(gf.predict_proba(X)[:, 1], ((1 - value[at]) + 0.75) / 2)


@pytest.mark.parametrize("H,W,D", [(17, 33, 17), (13, 47, 16), (30, 16, 5)])
def test_fused_classifier_at_tile_edges(gpu, H, W, D):
    from cbmv_b200.forest import FlatForest
    from cbmv_b200.forest_gpu import GpuForest
    from cbmv_b200.pipeline import StereoPipeline
    from conftest import FOREST_PATH, rand_pair
    gf = GpuForest(FlatForest.load(FOREST_PATH))
    pipe = StereoPipeline(gf)
    L, R = rand_pair(9, H, W, flat=True)
    X = pipe.features_at(L, R, D, torch.arange(H * W * D, device="cuda"))
    prob = torch.empty((H, W, D), device="cuda")
    pipe.run_rf(L, R, D, prob_out=prob)
    want = gf.predict_proba(X)[:, 0].to(torch.float32).view(H, W, D)
    assert torch.equal(prob, want)
