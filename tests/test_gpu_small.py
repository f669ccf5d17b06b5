"""Small worlds: the one-warp-per-slot density pass (csrc/pfs_small.cuh) and the
one-block sort (csrc/pfs_sort.cu) on both sides of their size limits, against the
oracle bit for bit (same terms, same order: no tolerance)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_oracle, load_package
from test_gpu_parity import _assert_bits_equal, _check_substep, _uniform_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 4096, 4097, 8192, 8193, 49152, 49153])
def test_small_world_substep(cuda_device, monkeypatch, n):
    monkeypatch.setenv("PFS_NEIGHBOR_SEARCH", "table")
    pfs, ora = load_package(), load_oracle()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=0.06)
    # walls, particles outside the box and a clump past the list rows
    pos[: n // 8, 0] = 0.0
    pos[n // 8: n // 6, 1] = 1.1
    rng = np.random.default_rng(n)
    k = min(n // 5, 600)
    pos[n - k:, :3] = 0.5 + rng.uniform(0.0, 0.03, (k, 3)).astype(np.float32)
    _check_substep(pfs, ora, p, pos, vel)


@pytest.mark.parametrize("n", [1, 500, 4097, 49152])
def test_small_world_fp16_equals_list_walk(cuda_device, n):
    """The FP16-cell form's small-world sums equal its grid search's."""
    pfs = load_package()
    p, pos, vel = _uniform_scene(pfs, n, seed=n, h=0.06)
    p.precision = pfs.PFS_FP16_CELL
    out = {}
    for search in (pfs.PFS_SEARCH_TABLE, pfs.PFS_SEARCH_GRID):
        with pfs.World(p, pos, vel) as w:
            w.set_shape(pfs.PFS_SHAPE_LIST, search)
            w.step(1)
            out[search] = w.read(density=True)
            assert w.device_error() == 0
    for key in ("pos", "vel", "density"):
        _assert_bits_equal(key, out[pfs.PFS_SEARCH_TABLE][key], out[pfs.PFS_SEARCH_GRID][key])


@pytest.mark.parametrize("n,bits", [(1, 1), (33, 8), (2048, 32), (2049, 17), (8191, 9), (8192, 32), (8193, 32)])
def test_small_sort_is_stable(cuda_device, n, bits):
    import torch
    pfs = load_package()
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[rng.random(n) < 0.3] = keys[0]
    d = torch.from_numpy(keys.view(np.int32)).cuda()
    out, perm = torch.empty_like(d), torch.empty_like(d)
    st = torch.cuda.current_stream().cuda_stream
    pfs.check(pfs.lib().pfs_sort_keys_static(d.data_ptr(), n, bits, out.data_ptr(), perm.data_ptr(), st), "sort")
    pfs.check(pfs.lib().pfs_sort_static_status(st), "status")
    want = np.argsort(keys, kind="stable")
    assert np.array_equal(perm.cpu().numpy().view(np.uint32), want.astype(np.uint32))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), keys[want])
