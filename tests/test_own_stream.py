"""A pipeline on a stream of its own: the device copies a call makes of host
or converted inputs are ordered before that stream's work and keep their
memory until it has passed them; results for the host wait for it."""
import numpy as np
import pytest


class _Stream:
    def __init__(self, handle):
        self.cuda_stream, self.waits = handle, []

    def wait_stream(self, other):
        self.waits.append(other.cuda_stream)


class _Tensor:
    def __init__(self, a):
        self.a, self.shape, self.on = a, a.shape, []

    def dim(self):
        return self.a.ndim

    def data_ptr(self):
        return id(self.a)

    def record_stream(self, s):
        self.on.append(s.cuda_stream)

    def contiguous(self):
        return self

    def cpu(self):
        return self

    def numpy(self):
        return self.a


@pytest.fixture
def calls(monkeypatch):
    """(the tensors made for a call, the current stream, the pipeline's)."""
    import torch
    from cbmv_b200 import _dev, _lib, pipeline
    cur, own, made = _Stream(7), _Stream(9), []

    def to_device(a, dtype):
        if isinstance(a, _Tensor) and a.a.dtype == dtype:
            return a, False
        made.append(_Tensor(np.asarray(a.a if isinstance(a, _Tensor) else a, dtype)))
        return made[-1], not isinstance(a, _Tensor)

    monkeypatch.setattr(_dev, "require_cuda", lambda: None)
    monkeypatch.setattr(_dev, "to_device", to_device)
    monkeypatch.setattr(_dev, "is_device", lambda a: isinstance(a, _Tensor))
    monkeypatch.setattr(_dev, "empty", lambda shape, dtype: _Tensor(np.zeros(shape, dtype)))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: cur)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda h: {9: own}[h])
    monkeypatch.setattr(_lib, "call", lambda *a: 0)
    monkeypatch.setattr(pipeline.StereoPipeline, "close", lambda self: None)
    monkeypatch.setattr(_lib, "default_params", lambda **k: _lib.cbmv_params())
    return made, cur, own


@pytest.mark.parametrize("cost", ["numpy", "float64", "own"])
def test_run_post_on_its_own_stream(calls, cost):
    from cbmv_b200.pipeline import StereoPipeline
    made, cur, own = calls
    img, vol = np.zeros((20, 30), np.uint8), np.zeros((20, 30, 4), np.float32)
    c = vol if cost == "numpy" else _Tensor(vol.astype(np.float64 if cost == "float64" else np.float32))
    StereoPipeline(stream=9).run_post(_Tensor(img), _Tensor(img), c)
    if cost == "own":
        assert made == [] and own.waits == [] and c.on == []  # the caller's own tensor: the caller's to order
    else:
        assert [t.on for t in made] == [[9]] and own.waits == [7]
    made.clear()
    StereoPipeline(stream=7).run_post(_Tensor(img), _Tensor(img), c)  # the current stream
    assert all(t.on == [] for t in made)


def test_host_results_wait_for_the_stream(calls):
    from cbmv_b200.pipeline import StereoPipeline
    made, cur, own = calls
    img = np.zeros((20, 30), np.uint8)
    out = StereoPipeline(stream=9).run_post(img, img, np.zeros((20, 30, 4), np.float32))
    assert isinstance(out, np.ndarray) and cur.waits == [9] and [t.on for t in made] == [[9]] * 3


@pytest.mark.gpu
def test_temporary_cost_outlives_the_call(gpu):
    """The stream is still busy when the call returns and its temporary cost
    is dropped; what is allocated next on torch's stream must not take it."""
    import torch
    from cbmv_b200.pipeline import StereoPipeline
    from conftest import rand_pair
    H, W, D = 64, 90, 32
    L, R = (torch.from_numpy(a).cuda() for a in rand_pair(2, H, W))
    cost = np.random.default_rng(0).random((H, W, D)).astype(np.float32)
    want = StereoPipeline().run_post(L, R, cost)
    s = torch.cuda.Stream()
    pipe = StereoPipeline(stream=s.cuda_stream)
    assert torch.equal(torch.from_numpy(pipe.run_post(L.cpu().numpy(), R.cpu().numpy(), cost)).cuda(), want)
    for given in (cost, torch.from_numpy(cost).cuda().double()):
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            torch.cuda._sleep(100_000_000)
        got = pipe.run_post(L, R, given)
        junk = [torch.full((H, W, D), float("nan"), device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        del junk
