"""swap_axes and swap_axes_back over their forms (a few disparities, tiles,
whole runs of large volumes) and the edges between them: a permutation, so
equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,H,W", [(1, 1, 1), (1, 37, 41), (7, 5, 33), (13, 64, 31), (14, 9, 70), (15, 33, 65), (16, 31, 9),
                                   (33, 33, 31), (65, 50, 61), (33, 500, 759), (65, 431, 451), (70, 401, 449),
                                   (127, 301, 333), (130, 300, 331), (257, 200, 251), (36, 501, 701), (700, 3, 5)])
def test_swaps_are_permutations(gpu, D, H, W):
    from cbmv_b200 import libfeatextract as fte
    v = torch.rand((D, H, W), dtype=torch.float64, device="cuda")
    want = v.permute(1, 2, 0).contiguous()
    assert torch.equal(fte.swap_axes(v), want)
    assert torch.equal(fte.swap_axes_back(want), v)
