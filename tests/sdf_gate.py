"""Host side of the distance field's sign: whether a mesh's sign is spread
(mpm::sdf_prepare_host of the library), and what its limits look at."""
import ctypes

import numpy as np


def spreads(mpm, tris, nodes):
    prepare = getattr(mpm.lib, "_ZN3mpm16sdf_prepare_hostEPKfixPf")
    floats = getattr(mpm.lib, "_ZN3mpm14sdf_aux_floatsEi")
    prepare.restype, floats.restype = ctypes.c_bool, ctypes.c_size_t
    t = np.ascontiguousarray(tris, np.float32)
    aux = np.zeros(floats(ctypes.c_int(len(t))) + 4, np.float32)
    return prepare(ctypes.c_void_p(t.ctypes.data), ctypes.c_int(len(t)), ctypes.c_longlong(nodes), ctypes.c_void_p(aux.ctypes.data))


def sliver(tris):
    """The largest L (L / h)^2 of the triangles (longest edge L, height h)."""
    t = np.asarray(tris, np.float64).reshape(-1, 3, 3)
    longest = np.max([np.linalg.norm(t[:, (k + 1) % 3] - t[:, k], axis=1) for k in range(3)], axis=0)
    return float((longest ** 5 / (np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]) ** 2).sum(1)).max())


def tilted_box(extent, tilt, through):
    """A box tilted from the axes by the slopes `tilt`, whose upper face has the
    point a quarter along its first axis at `through`."""
    from mpm_b200 import scenes
    n = np.array([tilt[0], tilt[1], 1.0])
    n /= np.linalg.norm(n)
    u = np.array([1.0, 0.0, 0.0]) - n[0] * n
    u /= np.linalg.norm(u)
    v = np.cross(n, u)
    corners = scenes.box_mesh(extent, (0.0, 0.0, 0.0)).reshape(-1, 3).astype(np.float64)
    corners -= np.array([-0.25 * extent[0], 0.0, 0.5 * extent[2]])
    return (corners @ np.stack([u, v, n]) + np.asarray(through)).astype(np.float32).reshape(-1, 9)
