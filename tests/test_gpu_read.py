"""pfs_world_read into device buffers: all at once, some, off the 16-byte grid (the
copies' path) and mixed with host arrays give the bytes of a host read."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import load_package
from test_gpu_parity import _uniform_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 2049])
@pytest.mark.parametrize("where", ["dddkk", "d----", "-d---", "--d--", "mmm--", "dmd--", "hdd--", "ddhkk", "-----"])
def test_read_targets(cuda_device, n, where):
    import torch
    pfs = load_package()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=0.2)
    words = [4 * n, 4 * n, n, n, n]
    names = ["pos", "vel", "density", "keys", "perm"]
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        want = w.read(pos=True, vel=True, density=True, keys=True, perm=True)
        bufs, ptrs = [], []
        for kind, k in zip(where, words):
            if kind == "-":
                bufs.append(None)
                ptrs.append(None)
                continue
            if kind == "h":
                t = torch.zeros(k + 2, dtype=torch.int32)
            else:
                t = torch.zeros(k + 2, dtype=torch.int32, device="cuda")
            t = t[1:k + 1] if kind == "m" else t[:k]
            torch.cuda.synchronize()
            bufs.append(t)
            ptrs.append(ctypes.c_void_p(t.data_ptr()))
        pfs.check(pfs.lib().pfs_world_read(w.handle, *ptrs), "pfs_world_read")
        for name, t in zip(names, bufs):
            if t is not None:
                got = t.cpu().numpy().view(np.uint32)
                assert np.array_equal(got, np.ascontiguousarray(want[name]).reshape(-1).view(np.uint32)), name
