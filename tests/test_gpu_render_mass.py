"""Volumetric rendering of a negative particle mass (pfs_params_validate takes one)
against the oracle: the light grows, and an empty sample in its way is Inf * 0."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package
from test_gpu_render import _tanf, _view, _world_scene, f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass", [-20.0, -0.5, 0.0, 0.5])
def test_volumetric_of_any_mass(cuda_device, mass):
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _world_scene(pfs)
    p.particle_mass, p.dt = mass, 0.0  # the block stays where it is (its forces would scatter it)
    v = _view(pfs)
    W, H = 64, 48
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        st = w.read(pos=True, keys=True)
        img, lv = w.render_volumetric(v, W, H, with_light_volume=True)
    dmap = ora.density_map(p, st["pos"], st["keys"], v.density_cell_size)
    lv_want = ora.light_volume(p, dmap, v.light_step_size, np.array(v.dir_to_sun[:], np.float32))
    assert np.array_equal(lv.view(np.uint32), lv_want.view(np.uint32))
    cam = np.array(list(v.position) + list(v.forward) + list(v.right) + list(v.up), np.float32)
    with np.errstate(all="ignore"):
        want = ora.volumetric(p, dmap, lv_want, cam, _tanf(f32(0.5) * f32(v.fov)), v.step_size,
                              np.array(v.extinction[:], np.float32), W, H)
    assert np.isnan(want[..., :3]).any() == (mass == -20.0)
    # (the last bits of expf differ between device and host: test_gpu_render.py)
    np.testing.assert_allclose(img, want, rtol=1e-4, atol=1e-6, equal_nan=True)
