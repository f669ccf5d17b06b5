"""launches_per_substep against the kernels the profiler records."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _scene(pfs, n, substeps=1):
    p = pfs.make_params(1.9 * (0.5 / n) ** (1 / 3), 1000.0, 50.0, 0.05, dt=0.001 * substeps, substeps=substeps)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = np.random.default_rng(n).uniform(0.05, 0.85, (n, 3))
    return p, pos, vel


def _kernels(step):
    import torch
    from torch.profiler import ProfilerActivity, profile
    step()  # captures the graph
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        step()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return [n for n in names if not n.lower().startswith(("memset", "memcpy"))]


# full tables (table scan): small and large; few slots: the grid search
@pytest.mark.parametrize("n,shape", [(2047, None), (60000, None), (1 << 16, None), (9000, "PFS_SHAPE_LIST"),
                                     (9000, "PFS_SHAPE_SIMPLE"), (16384, "PFS_SHAPE_LIST")])
def test_world_launches(cuda_device, n, shape):
    pfs = load_package()
    with pfs.World(*_scene(pfs, n)) as w:
        if shape:
            w.set_shape(getattr(pfs, shape))

        def step():
            w.step(1)
            w.sync()

        assert len(_kernels(step)) == w.launches_per_substep()


@pytest.mark.parametrize("sizes", [(2048, 4096), (9000, 5000), (2048, 9000)], ids=["table", "grid", "mixed"])
def test_batch_launches(cuda_device, sizes):
    pfs = load_package()
    b = pfs.Batch(sum(sizes), len(sizes), pfs.PFS_FP32, 1)
    for n in sizes:
        b.add(*_scene(pfs, n))

    def step():
        b.step(1)
        b.sync()

    assert len(_kernels(step)) == b.info()["launches_per_substep"]
    b.close()
