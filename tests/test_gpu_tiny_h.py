"""kn = 0 at a smoothing length whose near-pressure slope overflows: the shader's 0 * Inf
is NaN in every particle with a neighbour, in the lists, the queues and the grid search."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package

pytestmark = pytest.mark.gpu


# 45 / (pi h^6) overflows from 5.9e-7 down, 15 / (pi h^6) (the near density) from 4.9e-7 down
@pytest.mark.parametrize("h", [7e-7, 5.5e-7])
@pytest.mark.parametrize("n", [513, 1000, 1024])  # 2 slots (grid search), 256, 1,024
def test_near_pressure_of_tiny_h(cuda_device, n, h):
    pfs, ora = load_package(), load_oracle()
    p = pfs.make_params(h, 1000.0, 1e-9, 1e-9, dt=1e-9, box_min=(0, 0, 0), box_max=(8 * h, 8 * h, 8 * h))
    p.particle_mass, p.near_pressure_multiplier = 1e-16, 0.0
    p.margin_predict = p.margin_integrate = 0.0
    rng = np.random.default_rng(n)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.5 * h, 7.5 * h, (n, 3))
    with pfs.World(p, pos, vel) as w:
        got = w.debug_substep()
    with np.errstate(all="ignore"):
        want = ora.substep(p, pos, vel, trace=True)[3]
    a, b = got["vel_force"], want["vel_force"]
    assert np.array_equal(got["near_density"].view(np.uint32), want["near_density"].view(np.uint32))
    assert np.isnan(b[:, :3]).any() == (h < 5.9e-7)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(b)
    assert np.array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32))
