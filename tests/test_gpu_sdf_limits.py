"""The spread sign (makeSDF, kernels.cu:282-300) on closed meshes just inside the
limits within which it is used: the thinnest triangles, the largest coordinates
and both together, tilted a little from the grid so that the nodes on the two
sides of a face stand closest, against the FP64 oracle.

Where the sign is spread, a distance of 0.01 or more may exceed the true one by
half of the 0.001 by which the spread's balls fall short of the distances."""
import numpy as np
import pytest

from sdf_gate import sliver, spreads, tilted_box

pytestmark = pytest.mark.gpu

SIZE = (48, 40, 44)


@pytest.mark.parametrize("tilt", [(0.0, 0.0), (0.004, 0.0), (0.011, -0.007), (0.03, 0.02)])
@pytest.mark.parametrize("extent, least, coord", [
    ((517.0, 88.0, 88.0), 1.9e4, 300.0),   # thin
    ((30.0, 1.2, 1.2), 1.85e4, 0.0),       # thin and small: both sides of the box in the grid
    ((1300.0, 900.0, 900.0), 0.0, 960.0),  # far
    ((1300.0, 368.0, 368.0), 1.75e4, 960.0),  # thin and far
])
def test_signs_at_the_limits(gpu_ok, mpm, oracle64, extent, least, coord, tilt):
    from mpm_b200 import scenes
    box = tilted_box(extent, tilt, (23.4, 19.3, 21.47))
    tris = np.ascontiguousarray(np.concatenate([box, scenes.uv_sphere(9.0, (300.0, 310.0, 290.0), 40, 24)]), np.float32)
    assert least <= sliver(tris) < 2e4 and coord <= np.abs(tris).max() <= 1024.0
    cfg = scenes._cfg(SIZE)
    assert spreads(mpm, tris, cfg.grid_number)
    with mpm.Engine(cfg) as eng:
        eng.init_sdf(tris)
        got = eng.get_sdf().astype(np.float64)
    want, wn = oracle64.make_sdf(cfg, tris.astype(np.float64))
    assert ((want < 0).any() and (want > 0).any())
    over = (np.abs(got) - np.abs(want))[np.abs(got) >= 0.01]
    assert over.max() <= 5e-4
    # A node within FP32's error of the mesh may fall on either side of it.
    tol = 1e-4 + 8 * 2.0 ** -24 * np.abs(tris).max()
    sure = (np.abs(wn - 0.5) >= 1e-3) & (np.abs(want) > tol)
    wrong = (np.signbit(got) != np.signbit(want)) & sure
    assert not wrong.any(), f"{int(wrong.sum())} nodes of the wrong sign"
