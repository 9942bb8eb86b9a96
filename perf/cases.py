"""The performance cases of this framework: the work its users have it do,
through its public entry points, on seeded synthetic stereo pairs.

A case is a dict of plain values; `kind` names the entry point and the sizes
are W x H pixels and D disparities.  Kinds:

  pair      StereoPipeline.run_mlp: images -> matching cost + disparity (the
            driver's call; `host` = images and disparity in host memory)
  forest    StereoPipeline.run_rf: the same with the random forest
  post      StereoPipeline.run_post: the post-processing of a saved cost volume
  batch     StereoBatch.run_mlp: pairs of uneven size as one graph launch
  emit      StereoPipeline.features_at: training samples of one pair
  train     MlpTrainer.gradients: forward + backward of one training batch
  matchers  the libmatchers drop-ins as the reference's driver calls them
            (test.py:122-138), float64 volumes in [H,W,D]
  rows      libfeatextract.features + GpuForest.predict_proba on a band of
            rows (the reference classifies its image in such bands, test.py:608-623)
  dropin    the post drop-ins in the order of the reference's
            __postprocessing_mem (test.py:341-449)

Everything `prepare` makes is made on the GPU from the seed: value-noise
textures with flat patches, slanted-plane disparities, a z-buffered right
view with sensor noise.
"""
import functools
import math
import os
import random

import numpy as np
import torch
import torch.nn.functional as nnf

from cbmv_b200 import _lib, libfeatextract, libmatchers, post
from cbmv_b200.batch import StereoBatch
from cbmv_b200.forest import FlatForest
from cbmv_b200.forest_gpu import GpuForest
from cbmv_b200.mlp import GpuMlp, MlpParams, MlpTrainer, input_stats
from cbmv_b200.pipeline import StereoPipeline

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
NETS = {"gelu": os.path.join(GOLDEN, "mlp_gelu_694x554.npz"), "relu": os.path.join(GOLDEN, "mlp_694x554.npz")}
SENTINEL = 2147483647.0


def listed():
    return [
        # the smallest call: a thumbnail from host arrays, where launches and copies are the time
        {"name": "pair_96x64_host", "kind": "pair", "W": 96, "H": 64, "D": 16, "act": "gelu", "prec": "f16",
         "host": True, "interp": False},
        # an odd size with a disparity count that is no multiple of 4, bfloat16 operands, the left-right check
        {"name": "pair_451x319_d70_bf16_interp", "kind": "pair", "W": 451, "H": 319, "D": 70, "act": "gelu",
         "prec": "bf16", "host": False, "interp": True},
        # the benchmark's pair, with the cost volume kept as --saveCostVolume does
        {"name": "pair_694x554_d128", "kind": "pair", "W": 694, "H": 554, "D": 128, "act": "gelu", "prec": "f16",
         "host": False, "interp": False},
        # a large pair of the larger-configuration tests, with the ReLU network
        {"name": "pair_1482x994_d256_relu", "kind": "pair", "W": 1482, "H": 994, "D": 256, "act": "relu",
         "prec": "f16", "host": False, "interp": False},
        # the forest path on the benchmark's pair: the classifier that judges the network
        {"name": "forest_694x554_d128", "kind": "forest", "W": 694, "H": 554, "D": 128},
        # post-processing of a cost volume loaded from disk (--loadCostVolume), with the left-right check
        {"name": "post_901x600_d192_interp", "kind": "post", "W": 901, "H": 600, "D": 192, "interp": True},
        # several pairs of uneven size in one graph launch
        {"name": "batch_6_uneven", "kind": "batch", "n": 6, "sizes": 4000, "streams": 4, "act": "gelu"},
        # emission of the network's training samples, one pair of its training set
        {"name": "emit_694x554_d128", "kind": "emit", "W": 694, "H": 554, "D": 128, "n": 100000},
        # the trainer's batch
        {"name": "train_8192", "kind": "train", "batch": 8192, "act": "gelu"},
        # the reference's driver over the drop-in modules: matchers, classified row bands, post
        {"name": "matchers_694x554_d128", "kind": "matchers", "W": 694, "H": 554, "D": 128},
        {"name": "rows_694x144_d128", "kind": "rows", "W": 694, "H": 144, "D": 128},
        {"name": "dropin_post_694x320_d128", "kind": "dropin", "W": 694, "H": 320, "D": 128},
    ]


# kind -> how often it is drawn, and the largest H*W*D of a drawn case
DRAWN = {"pair": (5, 2.4e8), "forest": (1, 4.0e7), "post": (1, 1.2e8), "batch": (1, 0), "emit": (1, 5.0e7),
         "train": (2, 0), "matchers": (2, 4.9e7), "rows": (1, 1.2e7), "dropin": (1, 3.0e7)}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(list(DRAWN), [w for w, _ in DRAWN.values()])[0]
    act = rng.choice(["gelu", "gelu", "relu"])
    if kind == "train":
        return {"kind": kind, "batch": 128 * _log_uniform(rng, 1, 256), "act": act}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(2, 6), "sizes": rng.randint(0, 10 ** 6),
                "streams": rng.choice([1, 2, 4]), "act": act}
    most = DRAWN[kind][1]
    while True:
        W, H, D = _log_uniform(rng, 64, 1500), _log_uniform(rng, 48, 1000), _log_uniform(rng, 12, 256)
        if rng.random() < 0.6:  # calibration files give such disparity counts
            D = max(16, D // 16 * 16)
        if W * H * D <= most and D <= W:
            break
    case = {"kind": kind, "W": W, "H": H, "D": D}
    if kind == "pair":
        case.update(act=act, prec=rng.choice(["f16", "f16", "bf16"]), host=rng.random() < 0.3,
                    interp=rng.random() < 0.25)
    elif kind == "post":
        case.update(interp=rng.random() < 0.5)
    elif kind == "emit":
        case.update(n=_log_uniform(rng, 1000, 200000))
    return case


# ------------------------------------------------------------------ inputs
def _scene(W, H, D, seed):
    """Left and right uint8 images and the left view's disparity (float32),
    as cbmv_b200.synth makes them, on the GPU."""
    g = torch.Generator("cuda").manual_seed(seed)
    r = random.Random(seed)

    def noise(*shape):
        return torch.rand(*shape, device="cuda", generator=g)

    img = torch.zeros(H, W, device="cuda")
    period, amp = max(W / 8.0, 2.0), 1.0
    for _ in range(4):
        lat = noise(1, 1, math.ceil(H / period) + 2, math.ceil(W / period) + 2)
        up = nnf.interpolate(lat, scale_factor=max(period, 1.0), mode="bicubic", align_corners=False)
        img += amp * up[0, 0, :H, :W]
        period, amp = max(period / 2.0, 1.0), amp * 0.5
    img -= img.min()
    img *= 255.0 / img.max()
    area = 0
    while area < 0.1 * H * W:
        h, w = min(r.randint(8, 64), H), min(r.randint(8, 64), W)
        y, x = r.randint(0, H - h), r.randint(0, W - w)
        img[y:y + h, x:x + w] = r.uniform(0, 255)
        area += h * w
    left = img.round().clamp(0, 255)
    yy, xx = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    gt = torch.zeros(H, W, device="cuda")
    best = torch.full((H, W), float("inf"), device="cuda")
    lo, hi = 1.0, max(2.0, 0.94 * (D - 3))
    for _ in range(12):
        cy, cx = r.uniform(0, H), r.uniform(0, W)
        plane = r.uniform(lo, hi) + r.uniform(-0.2, 0.2) * (xx - cx) + r.uniform(-0.2, 0.2) * (yy - cy)
        dist = (yy - cy) ** 2 + (xx - cx) ** 2
        gt = torch.where(dist < best, plane, gt)
        best = torch.minimum(best, dist)
    gt = gt.clamp(lo, hi)
    # right view: every left pixel lands on x - d, the nearer surface wins; small gaps take their neighbour's
    tx = (xx - gt).round().long()
    inside = (tx >= 0) & (tx < W)
    z = torch.full((H * W,), -1.0, device="cuda")
    z.scatter_reduce_(0, (yy * W + tx)[inside], gt[inside], "amax")
    z = z.view(H, W)
    for _ in range(2):
        z = torch.where(z < 0, torch.roll(z, 1, 1), z)
    src = (xx + z).clamp(0, W - 1)
    x0 = src.floor().long()
    fr = src - x0
    right = left.gather(1, x0) * (1 - fr) + left.gather(1, (x0 + 1).clamp(max=W - 1)) * fr
    right = torch.where(z < 0, 255.0 * noise(H, W), right)
    right = right + 2.0 * torch.randn(H, W, device="cuda", generator=g)
    return left.to(torch.uint8), right.round().clamp(0, 255).to(torch.uint8), gt


def _cost(gt, D, seed):
    """A matching cost [H,W,D] in [0,1] as a classifier gives it: low at the
    surface, a second dip somewhere else, noise."""
    g = torch.Generator("cuda").manual_seed(seed + 77)
    H, W = gt.shape
    d = torch.arange(D, device="cuda", dtype=torch.float32)
    decoy = D * torch.rand(H, W, 1, device="cuda", generator=g)
    c = 1 - 0.95 * torch.exp(-(d - gt[:, :, None]) ** 2 / 4)
    c -= 0.5 * torch.exp(-(d - decoy) ** 2 / 2)
    c += 0.1 * torch.randn(H, W, D, device="cuda", generator=g)
    return c.clamp_(0.001, 0.999)


def _samples(gt, D, n, seed):
    """n sample indices (y*W + x)*D + d, half at the surface, half elsewhere, and their labels."""
    g = torch.Generator("cuda").manual_seed(seed + 99)
    H, W = gt.shape
    p = torch.randint(H * W, (n,), device="cuda", generator=g)
    true = gt.reshape(-1)[p].round().long()
    d = torch.where(torch.arange(n, device="cuda") % 2 == 0, true,
                    torch.randint(D, (n,), device="cuda", generator=g)).clamp(0, D - 1)
    return p * D + d, ((d - gt.reshape(-1)[p]).abs() <= 1).float()


def _normalised(img):
    f = img.float()
    return ((f - f.mean()) / f.std(unbiased=False)).contiguous()


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [(r.randint(240, 720), r.randint(320, 1100), r.choice([64, 96, 128, 192])) for _ in range(case["n"])]


@functools.lru_cache(maxsize=None)
def _forest():
    return GpuForest(FlatForest.load(os.path.join(GOLDEN, "forest_694x554.npz")))


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "batch":
        shapes = _batch_sizes(case)
        scenes = [_scene(w, h, d, seed * 131 + i) for i, (h, w, d) in enumerate(shapes)]
        s.update(batch=StereoBatch(shapes, streams=case["streams"]), net=GpuMlp.load(NETS[case["act"]]),
                 L=[x[0] for x in scenes], R=[x[1] for x in scenes])
        return s
    if kind == "train":
        n = case["batch"]
        L, R, gt = _scene(320, 240, 128, seed)
        idx, y = _samples(gt, 128, n, seed)
        X = StereoPipeline().features_at(L, R, 128, idx)
        cap, mu, sd = input_stats(X.cpu().numpy())
        s.update(net=MlpTrainer(MlpParams.init(seed, cap, mu, sd, case["act"]), batch=n), X=X, y=y)
        return s
    W, H, D = case["W"], case["H"], case["D"]
    L, R, gt = _scene(W, H, D, seed)
    s.update(L=L, R=R)
    if kind == "pair":
        s.update(pipe=StereoPipeline(params=_lib.default_params(interpolate=int(case["interp"]))),
                 net=GpuMlp.load(NETS[case["act"]], precision=case["prec"]))
        if case["host"]:
            s.update(L=L.cpu().numpy(), R=R.cpu().numpy())
        else:
            s.update(prob=torch.empty(H, W, D, device="cuda"))
    elif kind == "forest":
        s.update(pipe=StereoPipeline(_forest()), prob=torch.empty(H, W, D, device="cuda"))
    elif kind == "post":
        s.update(pipe=StereoPipeline(params=_lib.default_params(interpolate=int(case["interp"]))),
                 cost=_cost(gt, D, seed))
    elif kind == "emit":
        s.update(pipe=StereoPipeline(), idx=_samples(gt, D, case["n"], seed)[0])
    elif kind == "rows":
        s.update(forest=_forest(), vols=_matchers(L, R, D))
    elif kind == "dropin":
        s.update(L=_normalised(L), R=_normalised(R), cost=_cost(gt, D, seed))
    return s


# ------------------------------------------------------------------ one pass
def _matchers(L, R, D):
    return [libmatchers.census(L, R, D, 11),
            libfeatextract.swap_axes(libmatchers.nccNister(L, R, D, 3)),
            libfeatextract.swap_axes(libmatchers.sadsob(libmatchers.sobel(L), libmatchers.sobel(R), D, 5)),
            libfeatextract.swap_axes(libmatchers.zsad(L, R, D, 5))]


def _gaussian(sigma):
    """The reference's __gaussian (test.py:108-118), its centre offset by one."""
    kr = math.ceil(sigma * 3)
    o = np.arange(-1, 2 * kr) - kr
    return np.exp(-(o[:, None] ** 2 + o[None, :] ** 2) / (2 * sigma * sigma)).astype(np.float32)


def _dropin(imL, imR, cost):
    H, W, D = cost.shape
    L, R = post.CUDA_float_array(imL), post.CUDA_float_array(imR)
    arms = torch.zeros(4, H, W, device="cuda")
    cl, cr = post.CUDA_float_array(arms), post.CUDA_float_array(arms)
    post.cross(L, cl, 6, 0.07)
    post.cross(R, cr, 6, 0.07)
    c, t = post.CUDA_double_array(cost), post.CUDA_double_array(cost)
    for _ in range(2):
        t.set_to_zero()
        post.sgm(L, R, c, t, None, 1.3, 10.0, 0.12, 1.4, 2.2, 3.0, -1)
        post.CUDA_divide_double(t, 4)
        post.CUDA_copy_double(t, c)
    post.swap_axis_back(c, t)
    post.CUDA_copy_double(t, c)
    for _ in range(4):
        post.cbca(cl, cr, c, t, -1)
        post.CUDA_copy_double(t, c)
    vol = c.t.view(D, H, W)
    # the reference's driver takes the argmin outside its modules (test.py:408-409)
    disp, tmp = post.CUDA_float_array(vol.argmin(0)), post.CUDA_float_array(arms[0])
    post.subpixel_enchancement(disp, c, tmp)
    post.CUDA_copy_float(tmp, disp)
    post.median2d(disp, tmp, 3)
    post.CUDA_copy_float(tmp, disp)
    post.mean2d(disp, tmp, _gaussian(2.2), 1.3)
    return vol, tmp.t.view(H, W)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "pair":
        if case["host"]:
            return {"disp": s["pipe"].run_mlp(s["net"], s["L"], s["R"], case["D"])}
        return {"disp": s["pipe"].run_mlp(s["net"], s["L"], s["R"], case["D"], prob_out=s["prob"]),
                "cost": s["prob"]}
    if kind == "forest":
        return {"disp": s["pipe"].run_rf(s["L"], s["R"], case["D"], prob_out=s["prob"]), "cost": s["prob"]}
    if kind == "post":
        return {"disp": s["pipe"].run_post(s["L"], s["R"], s["cost"])}
    if kind == "batch":
        return {"disp": s["batch"].run_mlp(s["net"], s["L"], s["R"])}
    if kind == "emit":
        return {"X": s["pipe"].features_at(s["L"], s["R"], case["D"], s["idx"])}
    if kind == "train":
        g, loss = s["net"].gradients(s["X"], s["y"])
        return {"grads": g, "loss": loss}
    if kind == "matchers":
        return {"volumes": _matchers(s["L"], s["R"], case["D"])}
    if kind == "rows":
        X = libfeatextract.features(*s["vols"])
        return {"X": X, "proba": s["forest"].predict_proba(X)}
    vol, disp = _dropin(s["L"], s["R"], s["cost"])
    return {"cost": vol, "disp": disp}


# ------------------------------------------------------------------ the least work
NET_FLOPS = 2 * (20 * 128 + 128 * 128 + 128 * 64 + 64)
TREES, DEPTH = 50, 17  # the committed forest: comparisons per (pixel, d) of a walk


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["batch"]
        return {"bytes": n * 21 * 4 + 4 * 27329 * 2, "flops": 3 * n * NET_FLOPS}
    if kind == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(6 * h * w for h, w, _ in sizes), "flops": NET_FLOPS * sum(h * w * d for h, w, d in sizes)}
    px = case["W"] * case["H"]
    V = px * case["D"]
    if kind == "pair":
        return {"bytes": 6 * px + (0 if case["host"] else 4 * V), "flops": NET_FLOPS * V}
    if kind == "forest":
        return {"bytes": 6 * px + 4 * V, "flops": TREES * DEPTH * V}
    if kind == "post":
        return {"bytes": 6 * px + 4 * V, "flops": (2 if case["interp"] else 1) * V * (2 * 4 * 8 + 4 * 22)}
    if kind == "emit":
        return {"bytes": 2 * px + case["n"] * 88, "flops": 4 * 2 * 3 * V}
    if kind == "matchers":
        return {"bytes": 2 * px + 32 * V, "flops": V * (8 + 18 + 50 + 100)}
    if kind == "rows":
        return {"bytes": 32 * V + 80 * V + 16 * V, "flops": V * (TREES * DEPTH + 20 * 5)}
    return {"bytes": 8 * px + 8 * V, "flops": V * (2 * 4 * 8 + 4 * 22)}


# ------------------------------------------------------------------ the same in 64 bits
def _shift(a, d, fill=0):
    """a[..., x - d] for every x, `fill` left of the image."""
    return a if d == 0 else nnf.pad(a, (d, 0), value=fill)[..., :a.shape[-1]]


def _box(a, w):
    """Sums over w x w windows centred on every pixel (whole windows only), else 0."""
    r = w // 2
    out = torch.zeros_like(a)
    H, W = a.shape[-2:]
    if H >= w and W >= w:
        acc = 0
        for i in range(w):
            for j in range(w):
                acc = acc + a[..., i:H - w + 1 + i, j:W - w + 1 + j]
        out[..., r:H - r, r:W - r] = acc
    return out


def _volumes64(L, R, D):
    """The four matching costs (matchers.cpp:24-512) as float64 [H,W,D]."""
    H, W = L.shape
    l, r = L.double(), R.double()
    x = torch.arange(W, device=l.device)
    y = torch.arange(H, device=l.device)[:, None]
    out = [torch.full((H, W, D), SENTINEL, dtype=torch.float64, device=l.device) for _ in range(4)]

    def put(m, d, w, v):
        c = w // 2
        ok = (y >= c) & (y < H - w + c) & (x >= c + d) & (x < W - w + c)
        out[m][:, :, d] = torch.where(ok, v, SENTINEL)

    def bits(a):  # bit k: the window's centre is below its k-th pixel
        p = nnf.pad(a, (5, 5, 5, 5))
        return torch.stack([a < p[i:i + H, j:j + W] for i in range(11) for j in range(11)])

    def sob(a):
        o = torch.zeros_like(a)
        if H > 3 and W > 3:
            col = a[:-2] + 2 * a[1:-1] + a[2:]
            o[1:H - 2, 1:W - 2] = (col[:, 2:] - col[:, :-2])[:H - 3, :W - 3]
        return o

    bl, br = bits(L.int()), bits(R.int())
    al, ar = _box(l, 3), _box(r, 3)
    cl, cr = 1 / (9 * _box(l * l, 3) - al * al).sqrt(), 1 / (9 * _box(r * r, 3) - ar * ar).sqrt()
    sl, sr = sob(l), sob(r)
    ml, mr = _box(l, 5) / 25, _box(r, 5) / 25
    for d in range(min(D, W)):
        put(0, d, 11, (bl != _shift(br, d)).sum(0).double())
        n = 9 * _box(l * _shift(r, d), 3) - al * _shift(ar, d)
        crd = _shift(cr, d)
        put(1, d, 3, torch.where(torch.isfinite(cl) & torch.isfinite(crd), -n * cl * crd, 1.0))
        put(2, d, 5, _box((sl - _shift(sr, d)).abs(), 5))
        dif, m = l - _shift(r, d), ml - _shift(mr, d)
        acc = torch.zeros_like(l)
        p = nnf.pad(dif, (2, 2, 2, 2))
        for i in range(5):
            for j in range(5):
                acc += (p[i:i + H, j:j + W] - m).abs()
        put(3, d, 5, acc)
    return out


EPS, SIGMA = (0.01, 1.01, 0.01, 0.01), (128.0, 0.02, 20000.0, 20000.0)


def _features64(vols, y0, y1):
    """The 20 features (test.py:521-595) of rows y0..y1-1, float64 [rows*W*D, 20]."""
    H, W, D = vols[0].shape
    x = torch.arange(W, device=vols[0].device)[:, None]
    d = torch.arange(D, device=vols[0].device)
    has = x + d < W
    f = [None] * 20
    for m, vol in enumerate(vols):
        c = vol[y0:y1]

        def conf(v, mn, den):
            dead = mn == SENTINEL
            ratio = (mn + EPS[m]) / (v + EPS[m])
            lik = torch.exp(-(v - mn) ** 2 / SIGMA[m]) / den
            return ratio.masked_fill(dead, 0), lik.masked_fill(dead, 0)

        def stats(v):
            mn = v.amin(2, keepdim=True).clamp(max=SENTINEL)
            return mn, torch.exp(-(v - mn) ** 2 / SIGMA[m]).sum(2, keepdim=True)

        f[m] = c
        f[4 + m], f[8 + m] = conf(c, *stats(c))
        at = (x + d).clamp(max=W - 1).expand(y1 - y0, W, D)
        mn, den = stats(torch.where(has, c.gather(1, at), vol[0, 0, 0]))
        back = (x - d).clamp(min=0).expand(y1 - y0, W, D)
        left = x >= d
        ratio, lik = conf(c, mn.expand(-1, -1, D).gather(1, back), den.expand(-1, -1, D).gather(1, back))
        f[12 + m], f[16 + m] = ratio.masked_fill(~left, 0), lik.masked_fill(~left, 0)
    return torch.stack([v.reshape(-1) for v in f], 1)


GELU = {"f16": (0.37451171875, -0.042694091796875, 0.0022716522216796875),
        "bf16": (0.373046875, -0.04296875, 0.00238037109375)}


def _activation(x, act, prec):
    """The hidden layers' activation and its derivative (include/cbmv.h, cbmv_mlp_set_activation)."""
    if act == "relu":
        return x.clamp(min=0), (x > 0).double()
    a, b, c = GELU[prec]
    u = x * x
    q = 0.5 + x * ((c * u + b) * u + a)
    d = q + x * ((5 * c * u + 3 * b) * u + a)
    return x * q.clamp(0, 1), torch.where(q <= 0, 0.0, torch.where(q >= 1, 1.0, d))


def _net(params, dev):
    v = {k: torch.from_numpy(np.array(a)).to(dev).double() for k, a in params.views().items()}
    return v, (v["W1"], v["W2"], v["W3"]), (v["b1"], v["b2"], v["b3"])


def _forward64(params, X, prec):
    v, Ws, bs = _net(params, X.device)
    a = [(torch.minimum(X, v["cap"]) - v["mu"]) * v["inv_sd"]]
    da = []
    for w, b in zip(Ws, bs):
        h, dh = _activation(a[-1] @ w.T + b, params.activation, prec)
        a.append(h)
        da.append(dh)
    return a, da, a[-1] @ v["w4"] + v["b4"]


def _gradients64(params, X, y):
    v, Ws, _ = _net(params, X.device)
    a, da, z = _forward64(params, X.double(), "f16")
    y = y.double()
    loss = nnf.binary_cross_entropy_with_logits(z, y)
    dz = (torch.sigmoid(z) - y) / len(y)
    tail = [a[3].T @ dz, dz.sum()[None]]
    back, g = dz[:, None] * v["w4"], []
    for k in (2, 1, 0):
        ds = back * da[k]
        g = [(ds.T @ a[k]).reshape(-1), ds.sum(0)] + g
        back = ds @ Ws[k]
    return torch.cat(g + tail), loss[None]


def _walk64(flat, X):
    """sklearn's predict_proba (float32 features against float64 thresholds)."""
    dev = X.device
    feat, thr = torch.from_numpy(flat.feature).to(dev).long(), torch.from_numpy(flat.threshold).to(dev)
    left, right = torch.from_numpy(flat.left).to(dev).long(), torch.from_numpy(flat.right).to(dev).long()
    value = torch.from_numpy(np.stack([flat.value0, flat.value1], 1)).to(dev)
    X = X.float().double()
    p = torch.zeros(len(X), 2, dtype=torch.float64, device=dev)
    for root in flat.roots.tolist():
        n = torch.full((len(X),), root, device=dev)
        while True:
            leaf = left[n] < 0
            if bool(leaf.all()):
                break
            below = X.gather(1, feat[n].clamp(min=0)[:, None])[:, 0] <= thr[n]
            n = torch.where(leaf, n, root + torch.where(below, left[n], right[n]))
        p += value[n]
    return p / flat.n_trees


def _arms64(im, L1=6, tau=np.float32(0.07)):
    """Cross arms (post.cu:336-396): end coordinates left, right, up, down."""
    H, W = im.shape
    out = []
    for ax, sgn in ((1, -1), (1, 1), (0, -1), (0, 1)):
        n = (H, W)[ax]
        pos = torch.arange(n, device=im.device)
        pos = (pos[None, :] if ax else pos[:, None]).expand(H, W)
        end, done = pos + sgn * L1, torch.zeros(H, W, dtype=torch.bool, device=im.device)
        for k in range(1, L1 + 1):
            q = pos + sgn * k
            off = (q < 0) | (q >= n)
            v = im.gather(ax, q.clamp(0, n - 1))
            stop = off | ((k > 1) & ((im - v).abs() >= float(tau)))
            end = torch.where(stop & ~done, q, end)
            done |= stop
        out.append(end)
    return out


def _sgm64(imL, imR, c):
    """One sgm call over the four scan directions (post.cu:178-333), direction -1, divided by 4."""
    H, W, D = c.shape
    dev = c.device
    tau, pi1, pi2, al, q1, q2 = float(np.float32(0.12)), 1.3, 10.0, 1.4, 2.2, 3.0
    p1, p2 = [pi1, pi1 / (q1 * q2), pi1 / q1], [pi2, pi2 / (q1 * q2), pi2 / q1]
    d = torch.arange(D, device=dev)
    total = torch.zeros_like(c)
    inf = float("inf")
    for k in range(4):
        horizontal, n = k < 2, W if k < 2 else H
        lines = torch.arange(H if horizontal else W, device=dev)
        prev = None
        for step in range(n):
            at = step if k in (0, 2) else n - 1 - step
            was = at - (1 if k in (0, 2) else -1)
            cost = c[:, at] if horizontal else c[at]
            if prev is None:
                cur = cost
            else:
                one = (imL[:, at] - imL[:, was] if horizontal else imL[at] - imL[was]).abs()[:, None]
                if horizontal:
                    x, xw = at - d, was - d
                    ok = ((x >= 0) & (xw >= 0)).expand(H, D)
                    two = (imR[:, x.clamp(min=0)] - imR[:, xw.clamp(min=0)]).abs()
                else:
                    x = lines[:, None] - d
                    ok = x >= 0
                    two = (imR[at][x.clamp(min=0)] - imR[was][x.clamp(min=0)]).abs()
                two = torch.where(ok, two, 10.0)
                low, high = (one < tau) & (two < tau), (one > tau) & (two > tau)

                def pick(p):
                    return torch.where(low, p[0], torch.where(high, p[1], torch.tensor(p[2], device=dev).double()))

                a, b = pick(p1), pick(p1)
                mn = prev.amin(1, keepdim=True)
                lo = nnf.pad(prev, (1, 0), value=inf)[:, :D] + (a / al if k == 2 else a)
                hi = nnf.pad(prev, (0, 1), value=inf)[:, 1:] + (b / al if k == 3 else b)
                best = torch.minimum(torch.minimum(prev, mn + pick(p2)), torch.minimum(lo, hi))
                cur = cost + best - mn
            prev = cur
            if horizontal:
                total[:, at] += cur
            else:
                total[at] += cur
    return total / 4


def _cbca64(al, ar, c):
    """One cbca pass (post.cu:399-450) on [D,H,W], direction -1."""
    D, H, W = c.shape
    x = torch.arange(W, device=c.device).expand(H, W)
    y = torch.arange(H, device=c.device)[:, None].expand(H, W)
    out = torch.empty_like(c)
    for d in range(D):
        r = [_shift(a, d, 0) for a in ar]
        s = torch.maximum(al[0], r[0] + d).clamp(-1, W - 1)
        t = torch.minimum(al[1], r[1] + d).clamp(0, W)
        t = torch.maximum(t, s + 1)
        acc = nnf.pad(c[d].cumsum(1), (1, 0))
        rows = nnf.pad((acc.gather(1, t) - acc.gather(1, s + 1)).cumsum(0), (0, 0, 1, 0))
        cnt = nnf.pad((t - s - 1).cumsum(0), (0, 0, 1, 0))
        top = torch.maximum(al[2], r[2])
        end = torch.minimum(al[3], r[3]).clamp(0, H)
        end = torch.maximum(end, top + 1)
        mean = (rows.gather(0, end) - rows.gather(0, top + 1)) / (cnt.gather(0, end) - cnt.gather(0, top + 1))
        out[d] = torch.where(x < d, c[d], mean)
    return out


def exact(case, seed):
    """Values for the costs, volumes, features, probabilities and gradients;
    a disparity (an argmin over near-equal costs) has none."""
    kind = case["kind"]
    if kind in ("batch", "post") or kind == "pair" and case["host"]:
        return None
    if kind == "train":
        s = prepare(case, seed)
        g, loss = _gradients64(s["net"].params(), s["X"], s["y"])
        return {"grads": g, "loss": loss}
    W, H, D = case["W"], case["H"], case["D"]
    if W * H * D > 6e7 or kind == "forest":
        return None
    L, R, gt = _scene(W, H, D, seed)
    if kind == "dropin":
        imL, imR = _normalised(L), _normalised(R)
        c = _cost(gt, D, seed).double()
        for _ in range(2):
            c = _sgm64(imL, imR, c)
        c = c.permute(2, 0, 1).contiguous()
        al, ar = _arms64(imL), _arms64(imR)
        for _ in range(4):
            c = _cbca64(al, ar, c)
        return {"cost": c, "disp": None}
    vols = _volumes64(L, R, D)
    if kind == "matchers":
        return {"volumes": vols}
    step = max(1, int(2e6 // (W * D)))
    bands = [(y, min(y + step, H)) for y in range(0, H, step)]
    if kind == "rows":
        X = torch.cat([_features64(vols, *b) for b in bands])
        return {"X": X, "proba": torch.cat([_walk64(_forest().flat, x) for x in X.split(4000000)])}
    if kind == "emit":
        idx = _samples(gt, D, case["n"], seed)[0]
        X = torch.empty(len(idx), 20, dtype=torch.float64, device="cuda")
        for a, b in bands:
            here = (idx >= a * W * D) & (idx < b * W * D)
            X[here] = _features64(vols, a, b)[idx[here] - a * W * D]
        return {"X": X}
    params = MlpParams.load(NETS[case["act"]])
    cost = [torch.sigmoid(-_forward64(params, _features64(vols, *b), case["prec"])[2]) for b in bands]
    return {"disp": None, "cost": torch.cat(cost).view(H, W, D)}
