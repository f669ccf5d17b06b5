"""The cell-grouped density pass of the grid search (csrc/pfs_cells.cuh) at the
edges of its blocks, stages and tables: bit-exact with the oracle in FP32 and
bit-identical to the table scan in the FP16-cell form (each sums the same terms
in the same order, so the tolerance is none)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package
from test_gpu_parity import _assert_bits_equal, _check_substep, _uniform_scene

pytestmark = pytest.mark.gpu


def _scene(pfs, name):
    n, h, clump = {
        "one_particle": (1, 0.3, 0),
        "tile_of_128_and_one": (1033, 0.5, 0),   # 8 cells, 129 each: two tiles per cell
        "single_cell_grid": (600, 2.0, 0),       # one cell holds the box
        "sparse_64_cell_blocks": (9001, 0.03, 0),
        "two_layers_a_stage": (12289, 0.09, 0),
        "one_layer_a_stage": (20001, 0.165, 0),  # 90 per cell
        "too_dense_for_a_stage": (20001, 0.25, 0),
        "cell_by_cell": (9001, 0.05, 900),       # a clump overflows its block's stage only
        "pile": (21001, 0.05, 12000),            # more than a block is tried with
        "few_slots": (4097, 0.08, 0),            # two table slots: every run repeats
        "coarse_buckets": (1537, 0.004, 0),      # more cells than the buffers hold
    }[name]
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=h)
    if clump:
        rng = np.random.default_rng(clump)
        pos[:clump, :3] = 0.5 + rng.uniform(0.0, 0.8 * h, (clump, 3)).astype(np.float32)
    return p, pos, vel


NAMES = ["one_particle", "tile_of_128_and_one", "single_cell_grid", "sparse_64_cell_blocks", "two_layers_a_stage",
         "one_layer_a_stage", "too_dense_for_a_stage", "cell_by_cell", "pile", "few_slots", "coarse_buckets"]


@pytest.mark.parametrize("name", NAMES)
def test_cells_match_oracle(cuda_device, monkeypatch, name):
    pfs, ora = load_package(), load_oracle()
    monkeypatch.setenv("PFS_NEIGHBOR_SEARCH", "grid")
    _check_substep(pfs, ora, *_scene(pfs, name))


@pytest.mark.parametrize("name", NAMES)
def test_cells_fp16_equals_table_scan(cuda_device, monkeypatch, name):
    pfs = load_package()
    p, pos, vel = _scene(pfs, name)
    p.precision = pfs.PFS_FP16_CELL
    got = {}
    for mode in ("table", "grid"):
        monkeypatch.setenv("PFS_NEIGHBOR_SEARCH", mode)
        with pfs.World(p, pos, vel) as w:
            w.step(1)
            got[mode] = w.read(density=True)
            assert w.device_error() == 0
    for k in ("pos", "vel", "density"):
        _assert_bits_equal(k, got["grid"][k], got["table"][k])


def test_cells_on_faces(cuda_device, monkeypatch):
    """A lattice of spacing h: every particle on a cell face goes to the
    one-particle pass, its jittered neighbours do not."""
    pfs, ora = load_package(), load_oracle()
    monkeypatch.setenv("PFS_NEIGHBOR_SEARCH", "grid")
    h = 0.0625
    n = 4097
    side = 17
    idx = np.arange(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, 0], pos[:, 1], pos[:, 2] = idx % side * h, idx // side % side * h, idx // side ** 2 * h
    rng = np.random.default_rng(3)
    pos[::2, :3] += rng.uniform(-0.3 * h, 0.3 * h, (len(pos[::2]), 3)).astype(np.float32)
    p = pfs.make_params(h, 1000.0, 250.0, 0.03, gravity=(0, 0, 0), dt=1.0 / 240.0, box_max=(1.0625, 1.0625, 1.0625))
    _check_substep(pfs, ora, p, pos, np.zeros((n, 4), np.float32))


@pytest.mark.parametrize("seed", [12008, 11014, 11002])
def test_cells_pairs_on_the_cut(cuda_device, seed):
    """Dense enough that some pairs lie within an ulp of d = h, where a test
    that rounds otherwise than the reference's (a fused distance) takes or
    leaves one; its density term vanishes there, its force term does not."""
    pfs = load_package()
    from pfs_b200 import scenes
    sc = scenes.dam_break(72316, seed=seed, h=0.03802699223160744)
    out = {}
    for search in (pfs.PFS_SEARCH_TABLE, pfs.PFS_SEARCH_GRID):
        with pfs.World(sc.params, sc.pos, sc.vel) as w:
            w.set_shape(pfs.PFS_SHAPE_LIST, search)
            out[search] = w.debug_substep()
            assert w.device_error() == 0
    for k in ("density", "near_density", "vel_force"):
        _assert_bits_equal(k, out[pfs.PFS_SEARCH_GRID][k], out[pfs.PFS_SEARCH_TABLE][k])


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("n", [33, 12289])
def test_force_records_change_nothing(cuda_device, monkeypatch, n, fast):
    """The force pass reads a neighbour as one 32-byte record in a world created for
    the grid search, as three parts in one that comes to it later: the same bits."""
    pfs = load_package()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=0.12)
    if fast:
        p.precision = pfs.PFS_FP32_FAST
    out = {}
    for mode in ("table", "grid"):
        monkeypatch.setenv("PFS_NEIGHBOR_SEARCH", mode)
        with pfs.World(p, pos, vel) as w:
            w.set_shape(pfs.PFS_SHAPE_FLAT, pfs.PFS_SEARCH_GRID)
            w.step(2)
            out[mode] = w.read(pos=True, vel=True, density=True)
            assert w.device_error() == 0
    for k in ("pos", "vel", "density"):
        _assert_bits_equal(k, out["grid"][k], out["table"][k])
