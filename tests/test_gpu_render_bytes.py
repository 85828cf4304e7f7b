"""The renderer's 8-bit image against its float image (the framebuffer's
conversion of screen.frag's colour), and the splat's depth under any order of
the particles (the depth test keeps the nearest fragment, ssf_depth.frag)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (33, 7), (250, 131)])
@pytest.mark.parametrize("n", [0, 1, 257, 20_000])
def test_bytes_and_order(gpu_ok, mpm, size, n):
    import torch
    rng = np.random.default_rng(n + size[0])
    pos = (np.array([10.0, 8.0, 4.0]) + rng.random((n, 3)) * np.array([24.0, 20.0, 30.0])).astype(np.float32)
    seen = []
    for order in (slice(None), slice(None, None, -1), rng.permutation(n)):
        d = torch.from_numpy(pos[order].copy()).cuda()
        with mpm.Renderer((48, 40, 44), *size, light_dir=(0.1, 0.2, 1.0)) as r:
            r.render_device(d.data_ptr() if n else 0, n)
            f, b = r.image()
            seen.append((r.depth(0), f, b))
    for depth, f, b in seen:
        # (a 1 x 1 image has no neighbour to take a normal from: NaN, byte 0)
        assert np.array_equal(depth, seen[0][0]) and np.array_equal(f, seen[0][1], equal_nan=True)
        assert np.array_equal(b, seen[0][2])
    f = np.where(np.isnan(f), np.float32(0), f)
    want = np.floor(np.clip(f, np.float32(0), np.float32(1)) * np.float32(255) + np.float32(0.5)).astype(np.uint8)
    assert np.array_equal(b, want)
