"""The density map's flat walk (k_map_flat, csrc/pfs_density_map.cu) at the edges of
its blocks and range words, and the light volume on both sides of the quick division
(box_size, csrc/pfs_render.cu), against the oracle, bit for bit (the same operations
in the same order, so the tolerance is none)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package
from test_gpu_parity import _uniform_scene
from test_gpu_render import _view, _world_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,factor,clump", [
    (1, 0.3, 1.0, 0),        # one slot: every voxel's 27 runs are the one particle
    (2, 0.3, 7.0, 0),        # one voxel: a block of one
    (128, 0.2, 1.3, 0),      # ragged last block
    (4096, 0.06, 1.0, 126),  # range words of 127 and 128 particles
    (4096, 0.06, 1.0, 127),
    (8192, 0.05, 1.0, 5000), # more words than a column holds
    (4096, 0.05, 0.4, 0),    # several voxels a cell
    (8192, 0.05, 2.3, 0),    # cells without a voxel
])
def test_map_flat_matches_oracle(cuda_device, n, h, factor, clump):
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=h)
    if clump:
        rng = np.random.default_rng(clump)
        pos[:clump, :3] = 0.5 + rng.uniform(0.0, 0.1 * h, (clump, 3)).astype(np.float32)
    cs = float(np.float32(np.float32(h) * np.float32(factor)))
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        st = w.read(pos=True, keys=True)
        got = w.density_map(cs)
        assert w.device_error() == 0
    want = ora.density_map(p, st["pos"], st["keys"], cs)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert n < 3 or np.count_nonzero(want) > 0


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 30, 2.0 ** 42])
def test_light_volume_at_box_sizes(cuda_device, scale):
    """Boxes of 12 to 24 units and of 2^30 times that divide by the box's size in the
    quick way, those of 2^42 times that by the division."""
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _world_scene(pfs, n=4096)
    p.volume = float(p.h) ** 2 * 0.05 * scale ** 2  # densities of order one
    p.h *= scale
    for a in range(3):
        p.box_max[a] *= scale
    pos[:, :3] *= np.float32(scale)
    v = _view(pfs)
    v.density_cell_size *= scale
    v.light_step_size *= scale
    v.step_size *= scale
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        st = w.read(pos=True, keys=True)
        _, lv = w.render_volumetric(v, 16, 12, with_light_volume=True)
        assert w.device_error() == 0
    dmap = ora.density_map(p, st["pos"], st["keys"], v.density_cell_size)
    want = ora.light_volume(p, dmap, v.light_step_size, np.array(v.dir_to_sun[:], np.float32))
    assert lv.shape == want.shape and np.count_nonzero(want) > 0
    assert np.array_equal(lv.view(np.uint32), want.view(np.uint32))
