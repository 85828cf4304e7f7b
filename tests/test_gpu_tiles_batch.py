"""The touched-tile grid update over a batch (gridUpdate, kernels.cu:144-196):
scenes looked up in shared memory (up to 64) and in the global table (beyond),
CTAs of eight tiles that cross from one scene into the next, after a number of
substeps that leaves tiles behind, against the FP64 oracle's next substep."""
import numpy as np
import pytest

from parity import assert_normwise, assert_state_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 64, 70])
def test_tiles_in_a_batch(gpu_ok, mpm, oracle64, count):
    from mpm_b200 import scenes
    made = []
    for k in range(count):
        cfg, st, tris = scenes.small_scene(60 + 13 * k, (9 + k % 5, 12, 10 + k % 3), seed=700 + k, obstacle=(k % 9 == 4),
                                           padding=1)
        st[3] += 1.5  # drifts: tiles are left behind
        made.append((cfg, st, tris))
    with mpm.Batch([m[0] for m in made]) as b:
        b.init_all([m[1] for m in made])
        for k, m in enumerate(made):
            if len(m[2]):
                b.init_scene_sdf(k, m[2])
        b.set_tuning(12, 128, 0)
        b.step(4)
        pick = sorted({0, 1, count // 2, count - 1, 4 if count > 4 else 0})
        start = [b.scene_buffer(k) for k in pick]
        sdf = [b.scene_sdf(k) for k in pick]
        b.step(1)
        got = [b.scene_buffer(k) for k in pick]
        grid = [b.scene_grid(k) for k in pick]
    for k, s0, f, g, q in zip(pick, start, sdf, got, grid):
        want, wgrid, _, _ = oracle64.substep(made[k][0], s0.astype(np.float64), f.astype(np.float64))
        assert_state_close(g, want, s0)
        assert_normwise("grid mass", q[0], wgrid[0])
        assert_normwise("grid velocity", q[1:4], wgrid[1:4])
