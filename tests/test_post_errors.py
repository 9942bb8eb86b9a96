"""The post drop-ins report their errors as CbmvError."""
import pytest


class _Array:
    ins, ptr = [20, 30, 8], 16


def test_sgm_out_of_memory(monkeypatch):
    import torch
    from cbmv_b200 import _lib, post

    def empty(*a, **k):
        raise torch.OutOfMemoryError("CUDA out of memory")

    monkeypatch.setattr(torch, "empty", empty)
    with pytest.raises(_lib.CbmvError, match="out of memory") as e:
        post.sgm(_Array, _Array, _Array, _Array, None, 1.3, 10.0, 0.12, 1.4, 2.2, 3.0, -1)
    assert e.value.code == -2
