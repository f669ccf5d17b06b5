"""Which kernel makes a density map: maps of small worlds and of tables of few slots, where
grouping by cell or the flat walk was several times slower than a thread per voxel, against
the time of larger work of the same kind; and what is left by blocks that do not fit."""
from __future__ import annotations

import time

import numpy as np
import pytest

from conftest import load_oracle, load_package

pytestmark = pytest.mark.gpu


def _world(pfs, n, h, fill, seed=0, clump=0):
    p = pfs.make_params(h, 1000.0, 1.0, 0.01, dt=1e-5, gravity=(0.0, 0.0, 0.0))
    p.particle_mass = 1.0 / n
    rng = np.random.default_rng(seed)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = 0.002 + 0.996 * fill ** (1 / 3) * rng.uniform(0.0, 1.0, (n, 3))
    pos[:clump, :3] = 0.5 + 0.6 * h * rng.uniform(0.0, 1.0, (clump, 3))
    w = pfs.World(p, pos, vel)
    w.step(1)
    w.sync()
    return p, w


def _time(w, cs):
    import torch
    out = torch.empty(int(np.prod(w.density_map(cs).shape)), device="cuda")
    best = float("inf")
    for _ in range(8):
        t = time.perf_counter()
        w.density_map_ptr(cs, out.data_ptr())
        best = min(best, time.perf_counter() - t)
    return best


# A thread per voxel takes about 41 + 4 (n / slots + particles a cell) us of so few voxels: 130 to
# 250 here (up to twice that is allowed); grouped by cell 610 to 810.
@pytest.mark.parametrize("n,h", [(666, 0.13), (739, 0.15), (293, 0.2), (1323, 0.11)])
def test_small_maps(cuda_device, n, h):
    pfs = load_package()
    slots = 2 ** bin(n - 1).count("1")
    p, w = _world(pfs, n, h, 0.5)
    with w:
        assert _time(w, float(np.float32(h * 0.8))) < 2e-6 * (41.0 + 4.0 * (n / slots + n * h ** 3 / 0.5)) + 5e-5


# every form of the rule, the blocks' stages and what they leave, against the oracle
@pytest.mark.parametrize("n,h,fill,factor,clump", [
    (9001, 0.04, 1.0, 0.4, 2000),    # a clump in few blocks: left at once
    (40001, 0.03, 0.3, 0.5, 6000),   # a clump among blocks for every thread block: cell by cell, then left
    (40001, 0.02, 0.05, 0.6, 0),     # 128 slots, thin
    (8002, 0.114, 1.0, 1.0, 0),      # a stage all but full
    (16385, 0.05, 1.0, 0.7, 0),      # two slots
    (40064, 0.13, 1.0, 0.9, 0),      # 2,048 slots, 88 a cell
    (16384, 0.03, 0.01, 0.8, 0),     # a full table, long runs
])
def test_routes_match_oracle(cuda_device, n, h, fill, factor, clump):
    pfs, ora = load_package(), load_oracle()
    p, w = _world(pfs, n, h, fill, seed=n, clump=clump)
    cs = float(np.float32(h * factor))
    with w:
        st = w.read(pos=True, keys=True)
        got = w.density_map(cs)
        again = w.density_map(cs)
        assert w.device_error() == 0
    want = ora.density_map(p, st["pos"], st["keys"], cs)
    assert np.count_nonzero(want) > 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(again.view(np.uint32), want.view(np.uint32))
