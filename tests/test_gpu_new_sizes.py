"""A state of another particle count captures only the graphs that its steps
launch, when they are launched: loading it takes at most half again as long as
loading one of the same count (three times as long with both single-substep
graphs captured on the way), and the steps after it are those of a new engine."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_load_of_another_count(gpu_ok, mpm):
    from mpm_b200 import scenes
    cfg = scenes._cfg((32, 32, 32))
    rng = np.random.default_rng(3)
    states = [scenes.pack_state((4 + 24 * rng.random((8000 + k, 3))).astype(np.float32)) for k in range(4)]

    def median(eng, sequence):
        took = []
        for st in sequence:
            eng.step(0)
            begin = time.perf_counter()
            eng.init(st)
            took.append(time.perf_counter() - begin)
            eng.step(4)
        return float(np.median(took))

    with mpm.Engine(cfg) as eng:
        eng.init(states[3])
        eng.step(4)
        same, other = [], []
        for _ in range(3):  # in turn: the host's noise hits both
            same.append(median(eng, [states[0]] * 12))
            other.append(median(eng, [states[k % 4] for k in range(12)]))
    assert min(other) <= 1.5 * min(same), (other, same)


@pytest.mark.parametrize("calls", [(1,), (4,), (5, 1), (1, 4), (2, 6, 3)])
def test_first_steps_of_another_count(gpu_ok, mpm, calls):
    from parity import assert_state_close
    from mpm_b200 import scenes
    cfg, a, tris = scenes.small_scene(1500, (20, 18, 22), seed=61, padding=1)
    _, b, _ = scenes.small_scene(1501, (20, 18, 22), seed=62, padding=1)
    with mpm.Engine(cfg) as eng:
        eng.init(b)
        eng.step(sum(calls))
        want = eng.get_buffer()
    with mpm.Engine(cfg) as eng:
        eng.init(a)
        eng.step(6)
        eng.init(b)
        for c in calls:
            eng.step(c)
        got = eng.get_buffer()
    assert_state_close(got, want.astype(np.float64), b, rtol=1e-4)
