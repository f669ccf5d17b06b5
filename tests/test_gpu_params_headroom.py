"""A grid-search world keeps its blocks of single cells through pfs_world_set_params with a
somewhat smaller h or larger box: the cell-grouped density pass is still launched, and the
results are those of a world created with the parameters."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["PFS_FP32", "PFS_FP16_CELL"])
@pytest.mark.parametrize("h_factor,box_factor", [(0.97, 1.0), (0.82, 1.0), (1.0, 1.2), (1.1, 1.0)])
def test_blocks_survive_new_parameters(cuda_device, h_factor, box_factor, precision):
    pfs = load_package()
    n = 60001  # 128 slots
    p = pfs.make_params((8.0 / n) ** (1 / 3), 1000.0, 50.0, 0.05, dt=0.0005, precision=getattr(pfs, precision))
    p.particle_mass = 1000.0 / n
    rng = np.random.default_rng(5)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.002, 0.998, (n, 3))
    q = p.copy()
    q.h = p.h * h_factor
    for a in range(3):
        q.box_max[a] = p.box_max[a] * box_factor
    with pfs.World(p, pos, vel) as w, pfs.World(q, pos, vel) as fresh:
        launches = w.launches_per_substep()
        w.step(1)
        w.set_params(q)
        assert w.launches_per_substep() == launches == fresh.launches_per_substep()
        w.write(pos, vel)
        w.step(1)
        fresh.step(1)
        got, want = w.read(density=True), fresh.read(density=True)
        for name in want:
            assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name
        assert w.device_error() == 0
