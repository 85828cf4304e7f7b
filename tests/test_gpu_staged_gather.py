"""G2P's staged gather (g2PTransfer, kernels.cu:199-280): CTAs whose particles
lie in one bin, cross into a second, into a third and a fourth, at the walls of
the grid and outside it, alone and across the scenes of a batch, for both CTA
sizes, against the FP64 oracle."""
import numpy as np
import pytest

from parity import assert_state_close

pytestmark = pytest.mark.gpu


def _scene(kind, seed):
    from mpm_b200 import scenes
    rng = np.random.default_rng(seed)
    size = (40, 21, 23)
    cfg = scenes._cfg(size, padding=1)
    hi = np.array(size, np.float64)
    if kind == "dense":  # 10-odd particles per cell: a CTA is a layer or two of one bin
        pos = 2.0 + rng.random((9001, 3)) * np.array([14.0, 9.0, 7.0])
    elif kind == "sparse":  # below one per cell: a CTA crosses many bins
        pos = 1.0 + rng.random((1500, 3)) * (hi - 2.0)
    elif kind == "columns":  # full bins next to bins of a few particles
        a = np.array([6.5, 2.5, 2.5]) + rng.random((1300, 3)) * np.array([7.9, 3.9, 3.9])
        b = np.array([14.5, 6.5, 2.5]) + rng.random((37, 3)) * np.array([15.9, 7.9, 7.9])
        pos = np.concatenate([a, b])
    else:  # walls: the stencil leaves the grid on every side; some particles reach no node
        pos = rng.random((2000, 3)) * hi
        pos[::11] = hi + 3.0 + rng.random((len(pos[::11]), 3))
        pos[::7, 0] = 0.25
        pos[::5, 1] = hi[1] - 0.3
    st = scenes.pack_state(pos.astype(np.float32))
    st[3:6] = rng.normal(0, 0.5, (3, len(pos)))
    st[6:15] = rng.normal(0, 0.2, (9, len(pos)))
    return cfg, st


@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("kind", ["dense", "sparse", "columns", "walls"])
def test_staged_gather(gpu_ok, mpm, oracle64, kind, block):
    cfg, st = _scene(kind, 3)
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        eng.set_tuning(g2p_block=block)
        eng.step(1)
        got = eng.get_buffer()
    st0 = oracle64.init_particles(cfg, st)
    want, _, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
    assert_state_close(got, want, st0)


def test_staged_gather_batch(gpu_ok, mpm, oracle64):
    made = [_scene(k, s) for k, s in (("columns", 5), ("walls", 6), ("sparse", 7), ("dense", 8))]
    with mpm.Batch([m[0] for m in made]) as b:
        b.init_all([m[1] for m in made])
        b.step(1)
        got = [b.scene_buffer(k) for k in range(len(made))]
    for (cfg, st), g in zip(made, got):
        st0 = oracle64.init_particles(cfg, st)
        want, _, _, _ = oracle64.substep(cfg, st0, np.full(cfg.grid_number, 1e15))
        assert_state_close(g, want, st0)
