"""The distance field's sign and distances on closed meshes at the edge of what
FP32 distances can carry (makeSDF, kernels.cu:282-300): long thin triangles and
large coordinates, against the FP64 oracle.

The sign has to hold wherever the winding number is not within 1e-3 of its
threshold and the node lies further from the mesh than the tolerance.  The
distances carry FP32's error on such triangles: a few units in the last place
of the coordinates plus up to 2e-8 L (L / h)^2 cells (numpy's FP32 against 64
bits over rotated boxes) for a longest edge L and a height h; twice that here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _turned(extent, through):
    """A turned box, one of whose faces has its middle at `through`."""
    from mpm_b200 import scenes
    tris = scenes.box_mesh(extent, (0.0, 0.0, -0.5 * extent[2]))
    a, b = 0.7, 0.4
    r = (np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]])
         @ np.array([[1, 0, 0], [0, np.cos(b), -np.sin(b)], [0, np.sin(b), np.cos(b)]]))
    return (tris.reshape(-1, 3).astype(np.float64) @ r.T + np.asarray(through)).astype(np.float32).reshape(-1, 9)


# A sphere of ordinary triangles outside the grid takes the mesh past the line
# below which every node has its own sum (5e7 node-triangle pairs).
@pytest.mark.parametrize("extent", [(30.0, 10.0, 6.0), (36.0, 4.0, 4.0), (36.0, 0.8, 0.8), (34.0, 34.0, 0.5), (900.0, 700.0, 21.0),
                                    (1500.0, 1200.0, 700.0), (4000.0, 3000.0, 900.0)])
def test_sign_on_slivers_and_large_coordinates(gpu_ok, mpm, oracle64, extent):
    from mpm_b200 import scenes
    size = (40, 37, 41)
    near = _turned(extent, (19.7, 18.4, 20.3))
    far = scenes.uv_sphere(9.0, (300.0, 310.0, 290.0), 32, 20)
    tris = np.ascontiguousarray(np.concatenate([near, far]), np.float32)
    assert len(tris) * max(int(np.prod(size)), 65536) > 5e7
    cfg = scenes._cfg(size)
    with mpm.Engine(cfg) as eng:
        eng.init_sdf(tris)
        got = eng.get_sdf().astype(np.float64)
    want, wn = oracle64.make_sdf(cfg, tris.astype(np.float64))
    t = near.reshape(-1, 3, 3).astype(np.float64)
    longest = np.max([np.linalg.norm(t[:, (k + 1) % 3] - t[:, k], axis=1) for k in range(3)], axis=0)
    n2 = (np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]) ** 2).sum(1)
    tol = 1e-4 + 8 * 2.0 ** -24 * np.abs(t).max() + 4e-8 * (longest ** 5 / n2).max()
    sure = (np.abs(wn - 0.5) >= 1e-3) & (np.abs(want) > tol)
    wrong = (np.signbit(got) != np.signbit(want)) & sure
    assert not wrong.any(), f"{int(wrong.sum())} nodes of the wrong sign"
    assert np.abs(np.abs(got) - np.abs(want)).max() <= tol
