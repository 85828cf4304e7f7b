"""Positions after a frame (changeFormat, kernels.cu:341-347) are the state's,
bit for bit: particle counts around the export kernel's CTA size, and scenes
that begin and end inside a CTA, an empty one among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_positions_are_the_states(gpu_ok, mpm, n):
    from mpm_b200 import scenes
    cfg, st, _ = scenes.small_scene(n, (16, 16, 16), seed=n)
    with mpm.Engine(cfg) as e:
        e.init(st)
        for _ in range(3):
            e.step(2)
            assert np.array_equal(e.get_positions(), e.get_buffer()[:3].T)


def test_positions_of_a_batch(gpu_ok, mpm):
    from mpm_b200 import scenes
    made = [scenes.small_scene(n, (16, 16, 16), seed=n)[:2] for n in (100, 300, 1, 255, 600)]
    made.insert(2, (made[0][0], np.zeros((26, 0), np.float32)))
    with mpm.Batch([m[0] for m in made]) as b:
        b.init_all([m[1] for m in made])
        b.step(3)
        for k, m in enumerate(made):
            want = b.scene_buffer(k)[:3].T if m[1].shape[1] else np.zeros((0, 3), np.float32)
            assert np.array_equal(b.scene_positions(k), want)
