"""The grid search's blocks of cells are sized from the initial state wherever it is: a world
created from device memory steps like one created from host memory."""
from __future__ import annotations

import ctypes
import time

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N = 300000  # 4,096 slots


def _scene(pfs, seed=0):
    p = pfs.reference_default()
    rng = np.random.default_rng(seed)
    pos, vel = np.zeros((N, 4), np.float32), np.zeros((N, 4), np.float32)
    pos[:, :3] = rng.uniform(np.array(p.box_min[:]) * 0.3, np.array(p.box_max[:]) * 0.3, (N, 3))
    vel[:, 2] = -100.0
    return p, pos, vel


def _from_device(pfs, p, pos, vel):
    import torch
    x, v = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    pfs.check(pfs.lib().pfs_world_create(ctypes.byref(p), len(pos), ctypes.c_void_p(x.data_ptr()),
                                         ctypes.c_void_p(v.data_ptr()), ctypes.byref(h)), "pfs_world_create")
    return h


def _time(pfs, h, pos, vel):
    """The fastest of eight steps and the state after it."""
    L, ptr = pfs.lib(), lambda a: a.ctypes.data_as(ctypes.c_void_p)
    out, best = np.empty_like(pos), float("inf")
    for _ in range(8):
        pfs.check(L.pfs_world_write(h, ptr(pos), ptr(vel)), "write")
        pfs.check(L.pfs_world_sync(h, 0), "sync")
        t = time.perf_counter()
        pfs.check(L.pfs_world_step(h, 1), "step")
        pfs.check(L.pfs_world_sync(h, 0), "sync")
        best = min(best, time.perf_counter() - t)
    pfs.check(L.pfs_world_read(h, ptr(out), None, None, None, None), "read")
    return best, out


# unsized, the step of a world from device memory took 6.9 ms against 2.5
def test_world_from_device_memory(cuda_device):
    pfs = load_package()
    p, pos, vel = _scene(pfs)
    with pfs.World(p, pos, vel) as w:
        host, want = _time(pfs, w.handle, pos, vel)
    h = _from_device(pfs, p, pos, vel)
    dev, got = _time(pfs, h, pos, vel)
    pfs.check(pfs.lib().pfs_world_destroy(h), "destroy")
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert dev < 1.5 * host, (dev, host)


@pytest.mark.parametrize("n", [1, 2, 3, 513, 4097, 9217])
def test_small_worlds_from_device_memory(cuda_device, n):
    pfs = load_package()
    p = pfs.make_params(0.1, 1000.0, 50.0, 0.05, dt=0.0005)
    rng = np.random.default_rng(n)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.1, 0.9, (n, 3))
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        want = w.read()["pos"]
    h = _from_device(pfs, p, pos, vel)
    pfs.check(pfs.lib().pfs_world_step(h, 1), "step")
    got = np.empty_like(want)
    pfs.check(pfs.lib().pfs_world_read(h, got.ctypes.data_as(ctypes.c_void_p), None, None, None, None), "read")
    pfs.check(pfs.lib().pfs_world_destroy(h), "destroy")
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
