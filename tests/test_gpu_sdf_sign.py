"""The distance field's two sign forms (makeSDF, kernels.cu:282-300) against the
FP64 oracle: closed meshes, whose sign spreads through the balls of the nodes'
distances, and the others, which sum the winding number at every node.

Tolerance as in the other SDF tests: 1e-4 cells wherever the winding number is
not within 1e-3 of the 0.5 threshold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _meshes():
    from mpm_b200 import scenes
    sphere = scenes.uv_sphere(8.0, (14.3, 13.8, 15.1), 20, 10)
    flip = lambda t: t.reshape(-1, 3, 3)[:, [0, 2, 1]].reshape(-1, 9).copy()
    return {
        # open: a hole, a lone triangle, an edge run through twice the same way
        "hole": ((29, 30, 33), sphere[17:]),
        "one_triangle": ((16, 17, 18), np.array([[2.5, 3.1, 4.2, 12.3, 5.0, 6.1, 6.2, 13.4, 9.9]], np.float32)),
        "one_flipped": ((29, 30, 33), np.concatenate([flip(sphere[:1]), sphere[1:]])),
        # closed: faces on grid nodes, turned inside out, one shape in another,
        # two shapes that cross, a plate thinner than a cell, a mesh outside
        "box_on_nodes": ((24, 20, 17), scenes.box_mesh((10.0, 8.0, 6.0), (12.0, 9.0, 8.0))),
        "inside_out": ((29, 30, 33), flip(sphere)),
        "nested": ((40, 40, 40), np.concatenate([scenes.uv_sphere(15.0, (19.6, 20.2, 20.1), 24, 12),
                                                 flip(scenes.uv_sphere(6.0, (18.1, 20.0, 21.3), 16, 8))])),
        "crossing": ((40, 33, 35), np.concatenate([scenes.uv_sphere(9.0, (14.2, 16.1, 17.3), 16, 9),
                                                   scenes.box_mesh((17.0, 6.3, 9.1), (22.4, 17.2, 18.1))])),
        "plate": ((33, 20, 31), scenes.box_mesh((25.0, 0.4, 22.0), (16.2, 9.7, 15.1))),
        "outside": ((20, 20, 20), scenes.uv_sphere(6.0, (31.0, 10.0, 10.0), 12, 6)),
        # sizes: one triangle short of a group of 32 and one over, one node
        "31_triangles": ((18, 18, 18), np.concatenate([sphere[:31]]) * np.float32(0.6)),
        "33_triangles": ((18, 18, 18), np.concatenate([sphere[:33]]) * np.float32(0.6)),
        "one_node": ((1, 1, 1), scenes.box_mesh((4.0, 4.0, 4.0), (0.5, 0.5, 0.5))),
        # degenerate triangles beside a closed mesh, and a needle
        "degenerate": ((29, 30, 33), np.concatenate([sphere, np.repeat(sphere[3:4, :3], 3, 0).reshape(1, 9)])),
        "needle": ((20, 20, 20), np.array([[3.2, 4.1, 5.3, 15.2, 4.1, 5.3, 15.2, 4.1001, 5.3]], np.float32)),
    }


def _split(tris):
    """Every triangle in four, at its edges' midpoints."""
    a, b, c = np.split(tris.reshape(-1, 9), 3, axis=1)
    h = np.float32(0.5)
    ab, bc, ca = (a + b) * h, (b + c) * h, (c + a) * h
    return np.concatenate([np.concatenate(q, 1) for q in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))])


# Few nodes and triangles are summed at every node whatever the mesh: split
# until the line (5e7 pairs, at least 65536 nodes counted) is passed.
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("name", sorted(["hole", "one_triangle", "one_flipped", "box_on_nodes", "inside_out", "nested",
                                         "crossing", "plate", "outside", "31_triangles", "33_triangles", "one_node",
                                         "degenerate", "needle"]))
def test_sdf_sign_forms(gpu_ok, mpm, oracle64, name, split):
    from mpm_b200 import scenes
    size, tris = _meshes()[name]
    tris = np.ascontiguousarray(tris, np.float32)
    while split and len(tris) * max(int(np.prod(size)), 65536) <= 5e7:
        tris = np.ascontiguousarray(_split(tris), np.float32)
    cfg = scenes._cfg(size)
    with mpm.Engine(cfg) as eng:
        eng.init_sdf(tris)
        got = eng.get_sdf()
    want, wn = oracle64.make_sdf(cfg, tris.astype(np.float64))
    ok = np.abs(wn - 0.5) >= 1e-3
    err = np.abs(got.astype(np.float64) - want)[ok]
    assert err.max() <= 1e-4, f"max SDF error {err.max():.3e} cells"
    # where the sign is in doubt, the distance still holds
    assert np.abs(np.abs(got.astype(np.float64)) - np.abs(want)).max() <= 1e-4
