"""P2G (kernels.cu:6-142) against the FP64 oracle: the Tait pressure for whole
powers up to eight, by steps without powf, and for every other power, through
powf; and cells of more particles than a lane holds indices for at a time."""
import numpy as np
import pytest

from parity import assert_normwise, assert_state_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [1.0, 2.0, 7.0, 8.0, 9.0, 2.5, 0.5, 0.0, -0.5, -1.0, -2.0, -7.0, -8.0, -9.0, -3.25])
def test_powers(gpu_ok, mpm, oracle64, gamma):
    from mpm_b200 import scenes
    cfg, st, _ = scenes.small_scene(3000, (17, 15, 19), seed=31, obstacle=False, gamma=gamma, compression=12.0, padding=1)
    with mpm.Engine(cfg) as e:
        e.init(st)
        e.step(2)
        start = e.get_buffer()
        e.step(1)
        got, grid = e.get_buffer(), e.get_grid()
    sdf = np.full(17 * 15 * 19, 1e6)
    J = np.linalg.det(start[15:24].T.reshape(-1, 3, 3).astype(np.float64))
    assert (J > 1.001).sum() > 100 and (J < 0.999).sum() > 100
    want, wgrid, _, _ = oracle64.substep(cfg, start.astype(np.float64), sdf)
    assert_state_close(got, want, start)
    assert_normwise("grid mass", grid[0], wgrid[0])
    assert_normwise("grid velocity", grid[1:4], wgrid[1:4])


@pytest.mark.parametrize("cap", [31, 32, 33, 64])
def test_index_windows(gpu_ok, mpm, oracle64, cap):
    """Cells of 1 to 150 particles, summed by one lane up to the cap."""
    from mpm_b200 import scenes
    cfg, st, _ = scenes.small_scene(2600, (17, 15, 19), seed=33, obstacle=False, padding=1)
    rng = np.random.default_rng(5)
    counts = [1, 30, 31, 32, 33, 34, 63, 64, 65, 66, 97, 150] + [20] * 97
    cells = rng.permutation(9 * 9 * 9)[:len(counts)]
    base = np.repeat(np.stack([cells % 9, cells // 9 % 9, cells // 81], 1) + 4, counts, axis=0)[:2600]
    st = st[:, :len(base)].copy()
    st[:3] = (base + 0.55 + 0.9 * rng.random(base.shape)).T
    with mpm.Engine(cfg) as e:
        e.init(st)
        e.set_tuning(12, 128, 256, cap)
        start = e.get_buffer()
        e.step(1)
        got, grid = e.get_buffer(), e.get_grid()
    want, wgrid, _, _ = oracle64.substep(cfg, start.astype(np.float64), np.full(17 * 15 * 19, 1e6))
    assert_state_close(got, want, start)
    assert_normwise("grid mass", grid[0], wgrid[0])
    assert_normwise("grid velocity", grid[1:4], wgrid[1:4])
