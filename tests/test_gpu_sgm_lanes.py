"""The SGM scan over every number of disparities per lane, aligned and not,
against the same float32 recursion in numpy: equal (one order of operations;
a minimum has none)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32
PI1, PI2, TAU, ALPHA, Q1, Q2 = F(1.3), F(10), F(0.12), F(1.4), F(2.2), F(3)


def _scan(imL, imR, c, k, s):
    """Path costs of scan direction k (0 right, 1 left, 2 down, 3 up)."""
    H, W, D = c.shape
    out = np.empty_like(c)
    p1, p2 = [PI1, PI1 / (Q1 * Q2), PI1 / Q1], [PI2, PI2 / (Q1 * Q2), PI2 / Q1]
    n = W if k < 2 else H
    dx, dy = ((1, 0), (-1, 0), (0, 1), (0, -1))[k]
    y, x = (np.arange(H), None) if k < 2 else (None, np.arange(W))
    d = np.arange(D)
    prev = None
    for t in range(n):
        at = t if k in (0, 2) else n - 1 - t
        yy = y if k < 2 else np.full(W, at)
        xx = np.full(H, at) if k < 2 else x
        cost = c[yy, xx]
        if prev is None:
            cur = cost.copy()
        else:
            d1 = np.abs(imL[yy, xx] - imL[yy - dy, xx - dx])[:, None]
            xm = xx[:, None] + d * s
            ok = (xm >= max(0, dx)) & (xm < min(W, W + dx))
            xc = np.where(ok, xm, max(0, dx))
            d2 = np.where(ok, np.abs(imR[yy[:, None], xc] - imR[yy[:, None] - dy, xc - dx]), F(10))
            cls = np.where((d1 < TAU) & (d2 < TAU), 0, np.where((d1 > TAU) & (d2 > TAU), 1, 2))
            a = [np.array([v / ALPHA if k == m else v for v in p1], F)[cls] for m in (2, 3)]
            b = np.array(p2, F)[cls]
            mn = prev.min(1, keepdims=True)
            inf = np.full((len(prev), 1), np.inf, F)
            best = np.minimum(prev, mn + b)
            best = np.minimum(best, np.hstack([inf, prev[:, :-1]]) + a[0])
            best = np.minimum(best, np.hstack([prev[:, 1:], inf]) + a[1])
            cur = cost + best - mn
        out[yy, xx] = prev = cur
    return out


@pytest.mark.parametrize("D", [1, 31, 33, 64, 70, 96, 130, 160, 192, 224, 300, 384, 400, 512, 700, 1024])
@pytest.mark.parametrize("direction", [-1, 1])
def test_sgm_equals_float32_model(gpu, D, direction):
    from cbmv_b200 import _lib
    rng = np.random.default_rng(D)
    H, W = (5, 37) if D % 2 else (7, 66)
    imL, imR = ((rng.integers(0, 12, (H, W)) * F(0.06)).astype(F) for _ in range(2))
    vol = rng.random((H, W, D)).astype(F)
    want = np.ones_like(vol) + (((_scan(imL, imR, vol, 0, direction) + _scan(imL, imR, vol, 1, direction)) +
                                 _scan(imL, imR, vol, 2, direction)) + _scan(imL, imR, vol, 3, direction))
    a, b = torch.from_numpy(imL).cuda(), torch.from_numpy(imR).cuda()
    buf = torch.empty(vol.size + 4, device="cuda")
    scratch = torch.empty(_lib.lib().cbmv_sgm_scratch_bytes(H, W, D), dtype=torch.uint8, device="cuda")
    for off in (0, 1):
        v = buf[off:off + vol.size].view(H, W, D)
        v.copy_(torch.from_numpy(vol))
        out = torch.ones((H, W, D), device="cuda")
        _lib.call("cbmv_sgm_scratch", a.data_ptr(), b.data_ptr(), v.data_ptr(), H, W, D, PI1, PI2, TAU, ALPHA, Q1, Q2,
                  direction, out.data_ptr(), scratch.data_ptr(), None)
        assert np.array_equal(out.cpu().numpy(), want), off
