"""Results read into pageable memory, large ones by several threads through
pinned slots, are those read into pinned memory in one copy: sizes on both
sides of the 8 and 16 MB lines, ranges that end inside a chunk, and reads of one
object from several threads at once."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(shape, dtype):
    import torch
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    return torch.empty(n, dtype=torch.uint8).pin_memory().numpy().view(dtype).reshape(shape)


@pytest.mark.parametrize("n", [80660, 161319, 161320, 300001])  # 26 planes: 8 MiB + 32 B, 16 MiB - 40 B, + 64 B, 31.2 MB
def test_state_and_positions(gpu_ok, mpm, n):
    from mpm_b200 import scenes
    cfg, st, _ = scenes.small_scene(n, (32, 32, 32), seed=3, obstacle=False)
    with mpm.Engine(cfg) as e:
        e.init(st)
        e.step(1)
        want = _pinned((26, n), np.float32)
        assert mpm.lib.mpm_get_state(e._h, want.ctypes.data) == 0
        for _ in range(2):  # the first read may allocate the slots
            assert np.array_equal(e.get_buffer().view(np.uint32), want.view(np.uint32))
        assert np.array_equal(e.get_positions(), want[:3].T)


def test_image(gpu_ok, mpm):
    import torch
    pos = (torch.rand(20000, 3, device="cuda") * 20 + 6).contiguous()
    r = mpm.Renderer((32, 32, 32), 1913, 1507)  # 34.6 MB and 8.6 MB
    r.render_device(pos.data_ptr(), 20000, torch.cuda.current_stream().cuda_stream)
    rgb, rgb8 = r.image()
    want, want8 = _pinned(rgb.shape, np.float32), _pinned(rgb8.shape, np.uint8)
    assert mpm.lib.mpm_renderer_get_image(r._h, ctypes.c_void_p(want.ctypes.data), ctypes.c_void_p(want8.ctypes.data)) == 0
    assert np.array_equal(rgb, want) and np.array_equal(rgb8, want8)


def test_threads(gpu_ok, mpm):
    from mpm_b200 import scenes
    cfg, st, tris = scenes.small_scene(2000, (189, 183, 181), seed=4)
    with mpm.Engine(cfg) as e:
        e.init(st)
        e.init_sdf(tris)
        want = e.get_sdf()
        got = [None] * 4

        def read(k):
            got[k] = e.get_sdf()

        ts = [threading.Thread(target=read, args=(k,)) for k in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for g in got:
            assert np.array_equal(g, want)
