"""pfs_world_read into a device buffer that is too short: refused, as the copies refuse it,
and nothing beyond the buffer is written.  The buffers are neighbours in one block of the
runtime's heap and all the test's own, so no store could leave mapped memory."""
from __future__ import annotations

import ctypes

import pytest

from conftest import load_package
from test_gpu_parity import _uniform_scene

pytestmark = pytest.mark.gpu

SIZE, COUNT = 4096, 128


@pytest.fixture
def heap(cuda_device):
    """COUNT buffers of SIZE bytes, and the first of eight that follow each other."""
    import torch
    torch.cuda.init()
    rt = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
    bufs = []
    for _ in range(COUNT):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(SIZE)) == 0
        assert rt.cudaMemset(p, 0x5a, ctypes.c_size_t(SIZE)) == 0
        bufs.append(p.value)
    bufs.sort()
    runs = [k for k in range(COUNT - 8) if all(bufs[k + j] == bufs[k] + j * SIZE for j in range(8))]
    assert runs, "the heap places small buffers apart"

    def content(p):
        out = (ctypes.c_uint8 * SIZE)()
        assert rt.cudaMemcpy(out, ctypes.c_void_p(p), ctypes.c_size_t(SIZE), 2) == 0
        return bytes(out)

    yield bufs, bufs[runs[0]], content
    for p in bufs:
        assert rt.cudaFree(ctypes.c_void_p(p)) == 0


@pytest.mark.parametrize("which", ["pos", "vel", "density"])
def test_short_buffer_is_refused(heap, which):
    pfs = load_package()
    bufs, target, content = heap
    n = 1025 if which == "density" else 1024  # 4,100 and 16,384 bytes
    p, pos, vel = _uniform_scene(pfs, n, seed=3, h=0.2)
    with pfs.World(p, pos, vel) as w:
        w.step(1)
        w.sync()
        args = [ctypes.c_void_p(target) if name == which else None for name in ("pos", "vel", "density")]
        assert pfs.lib().pfs_world_read(w.handle, *args, None, None) == pfs.PFS_ECUDA
        for q in bufs:
            assert content(q) == b"\x5a" * SIZE
        w.step(1)  # the world goes on
        w.read(density=True)
