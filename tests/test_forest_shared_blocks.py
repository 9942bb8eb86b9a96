"""cbmv_forest_create on blocks that several slots name as their child: each
block is laid out once, however many paths lead to it, and the walk reads it
there."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from test_forest import _walk

LEAF = 0x80000000


def _chain(n, seed=3):
    """One tree of n blocks, every slot of a block naming the next block (the
    last block: four leaves)."""
    rng = np.random.default_rng(seed)
    blocks = np.zeros((n, 8), np.uint32)
    blocks[:, 0:3] = rng.normal(size=(n, 3)).astype(np.float32).view(np.uint32)
    f = rng.integers(0, 20, (n, 3)).astype(np.uint32)
    blocks[:, 3] = f[:, 0] | f[:, 1] << 8 | f[:, 2] << 16
    blocks[:, 4:8] = np.arange(1, n + 1)[:, None]
    blocks[-1, 4:8] = LEAF | np.arange(4)
    return blocks, np.array([[0.1, 0.9], [0.3, 0.7], [0.6, 0.4], [0.8, 0.2]]), np.array([0, n], np.int32)


def _random_dag(n, n_leaves, seed):
    """Two trees whose blocks name arbitrary later blocks or leaves."""
    rng = np.random.default_rng(seed)
    ends = np.array([0, n // 3, n], np.int32)
    blocks = np.zeros((n, 8), np.uint32)
    blocks[:, 0:3] = rng.normal(size=(n, 3)).astype(np.float32).view(np.uint32)
    for k in range(n):
        end = ends[np.searchsorted(ends, k, "right")]
        f = rng.integers(0, 20, 3)
        f[1:][rng.random(2) < 0.2] = 0xFF
        if k + 1 == end and rng.random() < 0.5:
            f[0] = 0xFF
        blocks[k, 3] = f[0] | f[1] << 8 | f[2] << 16
        for s in range(4):
            if f[0] == 0xFF or f[1 + s // 2] == 0xFF:
                blocks[k, 4 + s] = rng.integers(n_leaves)
            elif k + 1 < end and rng.random() < 0.7:
                blocks[k, 4 + s] = rng.integers(k + 1, min(end, k + 4))
            else:
                blocks[k, 4 + s] = LEAF | rng.integers(n_leaves)
    p = rng.random(n_leaves)
    return blocks, np.stack([p, 1 - p], 1), ends


CHILD = """
import ctypes, resource, sys
sys.path[:0] = [%r, %r]
from cbmv_b200 import _lib
from test_forest_shared_blocks import _chain
L = _lib.lib()
blocks, leafv, offs = _chain(64)
h = ctypes.c_void_p()
resource.setrlimit(resource.RLIMIT_DATA, (2 << 30, 2 << 30))
rc = L.cbmv_forest_create(blocks.ctypes.data, 64, leafv.ctypes.data, 4, offs.ctypes.data, 1, 20, ctypes.byref(h))
assert rc == 0 or b"forest upload" in L.cbmv_last_error(), (rc, L.cbmv_last_error())
"""


def test_a_shared_block_is_laid_out_once():
    """64 blocks with 4^63 paths: laid out within a bounded memory, so that
    the call gets as far as the upload."""
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    subprocess.run([sys.executable, "-c", CHILD % (ROOT, os.path.join(ROOT, "tests"))], check=True, timeout=120, env=env)


NO_MEMORY = """
import ctypes, resource, sys
import numpy as np
sys.path.insert(0, %r)
from cbmv_b200 import _lib
L = _lib.lib()
n = 1 << 20
k = np.arange(n, dtype=np.int64)
blocks = np.zeros((n, 8), np.uint32)
blocks[:, 4:8] = np.where(4 * k[:, None] + np.arange(1, 5) < n, 4 * k[:, None] + np.arange(1, 5), 0x80000000)
leafv, offs, h = np.zeros((1, 2)), np.array([0, n], np.int32), ctypes.c_void_p()
data = sum(int(f.split()[1]) << 10 for f in open("/proc/self/status") if f.startswith("VmData"))
resource.setrlimit(resource.RLIMIT_DATA, (data + (16 << 20), data + (16 << 20)))
rc = L.cbmv_forest_create(blocks.ctypes.data, n, leafv.ctypes.data, 1, offs.ctypes.data, 1, 20, ctypes.byref(h))
assert rc == -3 and b"host memory" in L.cbmv_last_error(), (rc, L.cbmv_last_error())
"""


def test_exhausted_host_memory_is_an_error_code():
    """A million blocks (64 MB of entries) with 16 MB left: CBMV_ENOMEM, no
    C++ exception through the C boundary."""
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    subprocess.run([sys.executable, "-c", NO_MEMORY % ROOT], check=True, timeout=120, env=env)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: _chain(12), lambda: _random_dag(40, 9, 1), lambda: _random_dag(700, 60, 2)])
def test_walk_over_shared_blocks(gpu, make):
    """Leaves and probabilities of the blocks' own walk in numpy: equal."""
    import torch
    from cbmv_b200 import _lib
    blocks, leafv, offs = make()
    X = np.random.default_rng(0).normal(size=(997, 20)).astype(np.float32)
    want_p, want_leaves = _walk(blocks, leafv, offs, X)[:2]
    h = ctypes.c_void_p()
    _lib.call("cbmv_forest_create", blocks.ctypes.data, len(blocks), leafv.ctypes.data, len(leafv), offs.ctypes.data,
              len(offs) - 1, 20, ctypes.byref(h))
    x = torch.from_numpy(X).cuda()
    p = torch.empty(len(X), 2, dtype=torch.float64, device="cuda")
    leaves = torch.empty(len(X), len(offs) - 1, dtype=torch.int32, device="cuda")
    try:
        _lib.call("cbmv_forest_predict", h, x.data_ptr(), len(X), p.data_ptr(), leaves.data_ptr(), None)
        torch.cuda.synchronize()
    finally:
        _lib.lib().cbmv_forest_destroy(h)
    assert np.array_equal(leaves.cpu().numpy(), want_leaves)
    assert np.array_equal(p.cpu().numpy(), want_p)
