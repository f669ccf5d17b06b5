"""The density map's cell-grouped kernel (csrc/pfs_density_map.cu) at the edges of
its blocks, stages and tables, against the oracle, bit for bit (the same terms in
the same order, so the tolerance is none)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package
from test_gpu_parity import _uniform_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,factor,clump", [
    (4096, 0.06, 1.0, 0),      # a full table: the plain kernel
    (5121, 0.06, 1.0, 0),      # four slots
    (10113, 0.07, 0.8, 0),     # 512 slots: runs of 20
    (4097, 0.06, 1.0, 0),      # two slots: every run holds everybody
    (12289, 0.09, 0.5, 0),     # eight voxels a cell
    (12289, 0.09, 0.3, 0),     # 37 a cell: several tiles a block
    (12289, 0.09, 1.7, 0),     # cells without a voxel
    (20001, 0.165, 0.7, 0),    # one layer of one cell at a time
    (20001, 0.25, 0.9, 0),     # too dense for a stage: voxels walk their runs
    (9001, 0.05, 1.0, 1500),   # a clump overflows its block's stage
    (300, 0.4, 0.11, 0),       # a coarse grid, many voxels a cell
    (20000, 0.02, 4.5, 0),     # many more cells than voxels: the plain kernel
])
def test_map_cells_match_oracle(cuda_device, n, h, factor, clump):
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=h)
    if clump:
        rng = np.random.default_rng(clump)
        pos[:clump, :3] = 0.5 + rng.uniform(0.0, 0.8 * h, (clump, 3)).astype(np.float32)
    cs = float(np.float32(np.float32(h) * np.float32(factor)))
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        st = w.read(pos=True, keys=True)
        got = w.density_map(cs)
        assert w.device_error() == 0
    want = ora.density_map(p, st["pos"], st["keys"], cs)
    assert np.count_nonzero(want) > 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("shift", [-0.0625, 0.0, 0.0625])
def test_map_cells_between_empty_blocks(cuda_device, shift):
    """Small clumps at the faces and corners of blocks of 4 x 4 x 4 cells (within
    rounding of them and a step away) among empty blocks, and at the box's walls."""
    pfs, ora = load_package(), load_oracle()
    h, n = 0.06, 7937  # 32 slots
    p, pos, vel = _uniform_scene(pfs, n, seed=5, h=h)
    p.gravity[:] = (0.0, 0.0, 0.0)
    lo, hi = np.array(p.box_min[:]), np.array(p.box_max[:])
    rng = np.random.default_rng(9)
    faces = np.arange(0, int((hi - lo).min() / h), 4)
    spot = lo + h * (rng.choice(faces, (16, 3)) + shift)
    spot[::2] += h * rng.integers(0, 5, (8, 3))
    at = rng.integers(0, 16, n)
    jitter = rng.choice([0.0, 1e-7, -1e-7, 0.01 * h, -0.01 * h], (n, 3))
    pos[:, :3] = np.clip(spot[at] + jitter, lo + 1e-3, hi - 1e-3)
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        st = w.read(pos=True, keys=True)
        for factor in (0.5, 1.0):
            cs = float(np.float32(np.float32(h) * np.float32(factor)))
            got = w.density_map(cs)
            want = ora.density_map(p, st["pos"], st["keys"], cs)
            assert 0 < np.count_nonzero(want) < want.size // 2
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        assert w.device_error() == 0
