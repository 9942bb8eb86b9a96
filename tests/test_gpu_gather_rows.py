"""The features of few samples, formed from their own rows' statistics, equal
those formed from the whole image's, bit for bit: right pixels at every place
of a 32-pixel block, rows of one to many registers, disparities left of the
image, repeated samples."""
import numpy as np
import pytest
import torch

from conftest import rand_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,D", [(12, 12, 1), (13, 70, 5), (12, 75, 33), (13, 140, 128), (12, 97, 130), (13, 65, 263),
                                   (12, 60, 264), (12, 45, 600), (12, 13, 1024)])
def test_few_samples_equal_many(gpu, H, W, D):
    from cbmv_b200.pipeline import StereoPipeline
    L, R = rand_pair(H * W + D, H, W)
    rng = np.random.default_rng(D)
    n = H * W // 3  # the most that are formed from their own rows
    few = rng.integers(0, H * W * D, n)
    few[0], few[-1], few[n // 2] = 0, H * W * D - 1, few[0]
    pipe = StereoPipeline()
    own = pipe.features_at(L, R, D, few.astype(np.int64))
    many = pipe.features_at(L, R, D, np.concatenate([few, rng.integers(0, H * W * D, n + 2)]).astype(np.int64))
    one = pipe.features_at(L, R, D, few[:1].astype(np.int64))
    a, b = (v.cpu().numpy().view(np.int32) for v in (own, many[:n]))
    assert np.array_equal(a, b)
    assert torch.equal(one, own[:1])
