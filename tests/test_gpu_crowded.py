"""Small worlds whose particles are nearly all each other's neighbours take the flat walk (two
launches more: the spatial order), with the oracle's results; others one warp per slot."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package

pytestmark = pytest.mark.gpu


def _world(pfs, n, side, precision):
    p = pfs.make_params(0.1, 1000.0, 1e-3, 1e-4, dt=1e-6, gravity=(0.0, 0.0, 0.0), precision=precision)
    p.particle_mass = 1.0 / n
    rng = np.random.default_rng(n)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = 0.42 + side * rng.uniform(0.0, 1.0, (n, 3))
    return p, pos, vel


# n times particles per cell: 16,384^2 = 2.7e8 in one cell; 4,096^2 = 1.7e7
@pytest.mark.parametrize("precision", ["PFS_FP32", "PFS_FP16_CELL"])
@pytest.mark.parametrize("n,side,crowded", [(16384, 0.06, True), (4096, 0.06, False), (16384, 0.55, False)])
def test_route_of_crowded_small_worlds(cuda_device, n, side, crowded, precision):
    pfs = load_package()
    p, pos, vel = _world(pfs, n, side, getattr(pfs, precision))
    q, xpos, xvel = _world(pfs, 65536, 0.55, getattr(pfs, precision))
    sort = 2 if n > 8192 else 0  # launches of the sort beyond one
    with pfs.World(p, pos, vel) as w, pfs.World(q, xpos, xvel) as large:
        assert w.launches_per_substep() == large.launches_per_substep() - 2 + sort - (0 if crowded else 2)
        w.step(1)
        w.read()
        assert w.device_error() == 0


@pytest.mark.parametrize("n", [8192, 9000])
def test_crowded_world_matches_oracle(cuda_device, n):
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _world(pfs, n, 0.06, pfs.PFS_FP32)
    with pfs.World(p, pos, vel) as w:
        w.set_shape(pfs.PFS_SHAPE_FLAT, pfs.PFS_SEARCH_TABLE)
        got = w.debug_substep()
    want = ora.substep(p, pos, vel, trace=True)[3]
    for name in ("density", "near_density", "vel_force"):
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name
