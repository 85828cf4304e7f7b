"""An engine's asynchronous steps while another library captures a graph on a
stream of its own, in the mode that refuses allocations everywhere: the engine's
first steps of every kind (which capture its own graphs) and its 64th frame
(which pins a page) leave that capture intact, and both results hold."""
import numpy as np
import pytest

from parity import assert_state_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls, frames_before", [((1, 1), 0), ((4,), 0), ((5, 4), 0), ((1, 1, 1, 1), 61)])
def test_steps_beside_a_capture(gpu_ok, mpm, calls, frames_before):
    import torch
    from mpm_b200 import scenes
    cfg, st, tris = scenes.small_scene(900, (20, 18, 22), seed=71, padding=1)
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        eng.step(sum(calls))
        want = eng.get_buffer()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with mpm.Engine(cfg) as eng:
        eng.init(st)
        for _ in range(frames_before):
            eng.step(0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):  # global mode
            x += 1
            for c in calls:
                eng.step_async(c)
            x += 1
        eng.synchronize()
        got = eng.get_buffer()
        graph.replay()
        torch.cuda.synchronize()
    assert (x == 2).all()
    assert_state_close(got, want.astype(np.float64), st, rtol=1e-4)
