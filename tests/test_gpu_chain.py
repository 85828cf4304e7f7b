"""Substeps launched four at a time are the substeps launched one by one: every
count up to nine from either parity, with a count's remainder, stage timing in
between, and states of the same and of other sizes loaded over kept graphs."""
import numpy as np
import pytest

from parity import assert_state_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("count", [3, 4, 5, 8, 9])
def test_counts(gpu_ok, mpm, first, count):
    from mpm_b200 import scenes
    cfg, st, tris = scenes.small_scene(2000, (20, 18, 22), seed=51, padding=1)
    got, stats = [], []
    for chunks in ([first, count], [1] * (first + count)):
        with mpm.Engine(cfg) as e:
            e.init(st)
            e.init_sdf(tris)
            launches = e.stats()["kernel_launches"]
            for c in chunks:
                e.step(c)
            stats.append((e.stats()["substeps"], e.stats()["kernel_launches"] - launches - len([c for c in chunks])))
            got.append((e.get_buffer(), e.get_sort()[0], e.get_positions()))
    assert stats[0] == (first + count, stats[1][1])
    assert_state_close(got[0][0], got[1][0].astype(np.float64), st, rtol=1e-4)
    assert (got[0][1] != got[1][1]).mean() < 0.01  # Morton keys of the last substep's start: cell borders may round apart
    assert np.array_equal(got[0][2], got[0][0][:3].T)


def test_kept_graphs(gpu_ok, mpm):
    from mpm_b200 import scenes
    cfg, a, tris = scenes.small_scene(2000, (20, 18, 22), seed=52, padding=1)
    _, b, _ = scenes.small_scene(2000, (20, 18, 22), seed=53, padding=1)
    _, c, _ = scenes.small_scene(1100, (20, 18, 22), seed=54, padding=1)

    def fresh(st, n):
        with mpm.Engine(cfg) as e:
            e.init(st)
            e.init_sdf(tris)
            e.step(n)
            return e.get_buffer()

    with mpm.Engine(cfg) as e:
        e.init(a)
        e.init_sdf(tris)
        e.step(6)
        for st, n, tune, timing in ((b, 5, None, 0), (b, 5, (8, 256, 128), 0), (c, 6, None, 0), (a, 7, None, 3), (a, 7, None, 0)):
            e.init(st)
            if tune:
                e.set_tuning(*tune)
            e.set_stage_timing(timing)
            e.step(n)
            assert_state_close(e.get_buffer(), fresh(st, n).astype(np.float64), st, rtol=1e-4)
