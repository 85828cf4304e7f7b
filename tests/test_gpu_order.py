"""The particle ordering's launch forms (sort_by_key's role, engine.cu:92-102):
the bin scan around the scene size from which bins are summed in a launch of
their own, crowded cells handed to P2G's list, and a substep begun stage by
stage and given up."""
import numpy as np
import pytest

from parity import assert_normwise, assert_state_close

pytestmark = pytest.mark.gpu


# 2 bins; 1 chunk of 2048 bins; 4 chunks (the last scanned in one launch); 5 chunks.
@pytest.mark.parametrize("size", [(5, 6, 3), (64, 40, 48), (64, 96, 112), (64, 128, 128)])
def test_bin_scan_sizes(gpu_ok, mpm, oracle64, size):
    from mpm_b200 import scenes
    rng = np.random.default_rng(size[0] + size[1])
    cfg = scenes._cfg(size, padding=1)
    pos = 1.0 + rng.random((20_000, 3)) * (np.array(size) - 2.0)
    # every seventh particle in one corner cell: far past the cap of a lane
    pos[::7] = 1.5 + 0.5 * rng.random((len(pos[::7]), 3))
    st = scenes.pack_state(pos.astype(np.float32))
    st[3:6] = rng.normal(0, 0.5, (3, len(pos)))
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        eng.step(1)
        got, grid = eng.get_buffer(), eng.get_grid()
    st0 = oracle64.init_particles(cfg, st)
    want, wgrid, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
    assert_state_close(got, want, st0)
    assert_normwise("grid mass", grid[0], wgrid[0])
    assert_normwise("grid velocity", grid[1:4], wgrid[1:4])


# P2G's items shared out over 8, 4, 2 and 1 warps (27, 28, 56 and 112 bins are
# the first counts past each step); cells of 0 to 11 particles, so that some
# parts of an item are empty.
@pytest.mark.parametrize("bins", [1, 27, 28, 55, 56, 111, 112])
def test_item_parts(gpu_ok, mpm, oracle64, bins):
    from mpm_b200 import scenes
    rng = np.random.default_rng(bins)
    cfg = scenes._cfg((70, 30, 30), padding=1)
    pos = []
    for b in range(bins):  # bin (bx, by, bz): base cells 8 bx - 2 .. 8 bx + 5 and so on
        lo = np.array([8 * (1 + b % 7) - 2, 4 * (1 + b // 7 % 5) - 2, 4 * (1 + b // 35) - 2]) + 0.5
        cells = rng.integers(0, [8, 4, 4], (12, 3))
        for k, c in enumerate(cells):
            pos.append(lo + c + rng.random((k, 3)))
    pos = np.concatenate(pos).astype(np.float32)
    st = scenes.pack_state(pos)
    st[3:6] = rng.normal(0, 0.5, (3, len(pos)))
    st[6:15] = rng.normal(0, 0.2, (9, len(pos)))
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        eng.step(1)
        got, grid = eng.get_buffer(), eng.get_grid()
    st0 = oracle64.init_particles(cfg, st)
    want, wgrid, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
    assert_state_close(got, want, st0)
    assert_normwise("grid mass", grid[0], wgrid[0])
    assert_normwise("grid velocity", grid[1:4], wgrid[1:4])


@pytest.mark.parametrize("upto", [1, 2, 3])
def test_given_up_substep_leaves_nothing(gpu_ok, mpm, oracle64, upto):
    from mpm_b200 import scenes
    cfg, st, tris = scenes.small_scene(6000, (24, 24, 24), seed=9, obstacle=False)
    st[0:3, ::5] = 12.25  # a crowded cell
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        for _ in range(3):
            eng.substep_partial(upto)  # each starts anew
        eng.step(1)
        got, grid = eng.get_buffer(), eng.get_grid()
    st0 = oracle64.init_particles(cfg, st)
    want, wgrid, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
    assert_state_close(got, want, st0)
    assert_normwise("grid mass", grid[0], wgrid[0])
