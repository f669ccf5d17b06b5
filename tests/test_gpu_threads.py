"""Distinct worlds on distinct host threads: a dense and a sparse grid-search world,
whose density passes ask for different amounts of shared memory, are captured anew and
stepped side by side.  Every call succeeds, and the results are one thread's."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

ROUNDS = 300


def _world(pfs, frac, precision):
    """8,193 particles (two table slots: grid search) in a part of the box."""
    n = 8193
    p = pfs.reference_default()
    p.h, p.substeps, p.precision = 6.0, 2, precision
    rng = np.random.default_rng(7)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(np.array(p.box_min[:]) * frac, np.array(p.box_max[:]) * frac, (n, 3))
    return pfs.World(p, pos, vel), p, pos, vel


@pytest.mark.parametrize("precision", ["PFS_FP32", "PFS_FP16_CELL"])
def test_two_worlds_on_two_threads(cuda_device, precision):
    pfs = load_package()
    worlds = [_world(pfs, frac, getattr(pfs, precision)) for frac in (0.18, 0.9)]
    want = []
    for w, p, pos, vel in worlds:
        w.write(pos, vel)
        w.step(1)
        want.append(w.read(density=True))
    failures = []

    def run(w, p, pos, vel, ref):
        try:
            for k in range(ROUNDS):
                w.set_params(p)  # drops the graph: the next step captures it again
                w.write(pos, vel)
                w.step(1)
                if k % 50 == 0:
                    got = w.read(density=True)
                    for name in ref:
                        if not np.array_equal(got[name].view(np.uint32), ref[name].view(np.uint32)):
                            failures.append(name)
            w.sync()
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            failures.append(repr(e))

    threads = [threading.Thread(target=run, args=(*w, ref)) for w, ref in zip(worlds, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]
    for w, *_ in worlds:
        w.close()
