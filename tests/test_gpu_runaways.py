"""G2P beside runaway particles (g2PTransfer, kernels.cu:199-280; isInBounds,
common.cuh:212-218): positions at and beyond 2^31 and at infinity, whose stencil
bases saturate, in the CTA that stages the lowest layers of the grid, alone and
across the scenes of a batch.  They reach no node: each ends as it does in a
scene without any other particle, and the others end as if it were not there."""
import numpy as np
import pytest

from parity import assert_state_close

pytestmark = pytest.mark.gpu

FAR = [3e9, np.inf, 2147483648.0, 4294967296.0, 1e30, -3e9, -np.inf]


def _scene(axis, seed):
    """300 particles in the grid's lowest layers along `axis`, in one bin's
    columns, and one runaway per value of FAR along it."""
    from mpm_b200 import scenes
    cfg = scenes._cfg((24, 20, 22), padding=1)
    rng = np.random.default_rng(seed)
    pos = 6.5 + rng.random((300 + len(FAR), 3)) * np.array([7.9, 3.9, 3.9])
    pos[:, axis] = 0.6 + 2.0 * rng.random(len(pos))
    pos = pos.astype(np.float32)
    pos[300:, axis] = np.array(FAR, np.float32)
    st = scenes.pack_state(pos)
    st[3:6, :300] = rng.normal(0, 0.5, (3, 300))
    st[6:15, :300] = rng.normal(0, 0.2, (9, 300))
    return cfg, st


def _check(cfg, st, got, oracle64, alone):
    near = np.ascontiguousarray(st[:, :300])
    st0 = oracle64.init_particles(cfg, near)
    want, _, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
    assert_state_close(got[:, :300], want, st0)
    np.testing.assert_array_equal(got[:, 300:], alone)
    assert (got[3:6, 300:] == 0).all()


def _alone(mpm, cfg, st):
    with mpm.Engine(cfg) as eng:
        eng.init(np.ascontiguousarray(st[:, 300:]))
        eng.step(1)
        return eng.get_buffer()


@pytest.mark.parametrize("block", [128, 256])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_runaways(gpu_ok, mpm, oracle64, axis, block):
    cfg, st = _scene(axis, 11 + axis)
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        eng.set_tuning(g2p_block=block)
        eng.step(1)
        got = eng.get_buffer()
        assert eng.stats()["health"] == 3  # not finite, out of the grid
    _check(cfg, st, got, oracle64, _alone(mpm, cfg, st))


def test_runaways_in_a_batch(gpu_ok, mpm, oracle64):
    made = [_scene(axis, 21 + axis) for axis in (2, 0, 2, 1)]
    with mpm.Batch([m[0] for m in made]) as b:
        b.init_all([m[1] for m in made])
        b.step(1)
        got = [b.scene_buffer(k) for k in range(len(made))]
    for (cfg, st), g in zip(made, got):
        _check(cfg, st, g, oracle64, _alone(mpm, cfg, st))
