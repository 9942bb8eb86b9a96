"""The autotuner's cache: choices that were timed on other kernels are not reused."""
import hashlib
import json


def test_choices_for_earlier_kernels_are_not_reused(monkeypatch):
    import torch
    from cbmv_b200 import batch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "B200")
    shapes = [(64, 96, 16), (48, 64, 12)]
    before = hashlib.sha1(json.dumps(["B200", sorted(shapes)]).encode()).hexdigest()[:16]
    now = batch._signature(shapes)
    assert now != before and batch._signature(shapes[::-1]) == now
    monkeypatch.setattr(batch, "LAUNCH_SHAPES", batch.LAUNCH_SHAPES + 1)
    assert batch._signature(shapes) != now


def test_a_cached_choice_of_these_kernels_is_returned(monkeypatch, tmp_path):
    import torch
    from cbmv_b200 import batch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "B200")
    shapes = [(64, 96, 16)]
    path = tmp_path / "c.json"
    path.write_text(json.dumps({batch._signature(shapes): {"streams": 1, "ms": 1.0}}))
    assert batch.tune_batch(shapes, None, [], [], cache_path=str(path)) == {"streams": 1, "ms": 1.0, "cached": True}
