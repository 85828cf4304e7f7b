"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain numbers and texts; prepare() builds what a user's
program has in hand (scene, engine, weights, device arrays), run() is one pass
through the public entry points, exact() the same pass in 64-bit torch.  The
kinds:

  clip     a scene simulated from its start: the host state goes in
           (Engine.init), `frames` frames of SUBSTEPS substeps run one by one
           as a viewer's loop does, and the final state comes back
  batch    the same for a batch of independent scenes of uneven sizes
  learned  the same with learned 4 x DT large steps
  train    optimisation steps of the learned corrector
  sdf      the distance field of an obstacle mesh
  render   one frame of the headless fluid renderer, read back as an image
  sort     the stand-alone Morton key sort on device arrays
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "water-sim-cuda_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mpm_b200  # noqa: E402
from mpm_b200 import learned, scenes  # noqa: E402

# Physics: the benchmark configs as given, the same with gravity pulling -y and
# the Tait law resisting compression, and the config.txt defaults.
PHYSICS = {
    "bench": dict(padding=3, gravity=-0.3, dt=0.1, gamma=7.0, compression=10.0, substeps=4),
    "physical": dict(padding=3, gravity=0.3, dt=0.1, gamma=-7.0, compression=10.0, substeps=4),
    "default": dict(padding=2, gravity=9.81, dt=0.01, gamma=-2.0, compression=200.0, substeps=10),
}


def _clip(name, physics, size, water, obstacle, frames, resolution=0.5, read="end", **more):
    return dict(name=name, kind="clip", physics=physics, sx=size[0], sy=size[1], sz=size[2], water=water,
                obstacle=obstacle, frames=frames, resolution=resolution, read=read, **more)


def listed():
    return [
        # A small scene stepped frame by frame, its positions read every frame
        # (an interactive viewer or a game loop): latency and launches.
        _clip("clip_small_8k", "physical", (32, 32, 32), "sphere", "none", 25, read="frame", radius=6.2, cy=18.0),
        # The sphere-drop config: 113k particles in 64^3, no obstacle, gravity
        # pulling down.
        _clip("clip_sphere_drop", "physical", (64, 64, 64), "sphere", "none", 25, radius=15.0, cy=40.0),
        # An odd grid and a ragged box under the config.txt default physics.
        _clip("clip_ragged_default", "default", (97, 61, 83), "box", "sphere", 10, fx=0.47, fy=0.55, fz=0.9),
        # The dam-break config (2M particles, 128^3, torus) over 100 substeps:
        # from the block at rest to the first splash.
        _clip("clip_dam_break_2M", "physical", (128, 128, 128), "box", "torus", 25, fx=0.4667, fy=0.3084, fz=1.0),
        # The dam break's literal extents (5.2M particles).
        _clip("clip_dam_break_5M", "physical", (128, 128, 128), "box", "torus", 12, fx=0.4667, fy=0.8, fz=1.0),
        # The 256^3 config: three boxes of water, three obstacles, about 7M
        # particles in a mostly empty grid.
        _clip("clip_scale_256", "physical", (256, 256, 256), "boxes", "three", 12),
        # 64 independent scenes of uneven sizes in one batch.
        dict(name="batch_64", kind="batch", physics="physical", count=64, frames=10),
        # The learned large step with the shipped weights on the dam break.
        dict(name="learned_dam_break_2M", kind="learned", steps=12, fx=0.4667, fy=0.3084, fz=1.0),
        # The corrector's training at its batch size.
        dict(name="train_65536", kind="train", steps=50, batch=65536, samples=262144),
        # The dam break's obstacle on its grid.
        dict(name="sdf_torus_128", kind="sdf", sx=128, sy=128, sz=128, mesh="torus", seg_u=48, seg_v=24, size=25.0),
        # One rendered frame of the dam break at the viewer's window size.
        dict(name="render_2M", kind="render", n=1989120, width=1920, height=1600, grid=128),
        # The reference's particle sort as an operator on device arrays.
        dict(name="sort_2M", kind="sort", n=1989120, grid=128, static=False),
    ]


def _log(rng, lo, hi):
    return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))


def draw(rng):
    kind = rng.choice(["clip"] * 6 + ["batch", "learned", "train", "sdf", "sdf", "render", "sort", "sort"])
    if kind == "clip":
        physics = rng.choice(["bench", "physical", "physical", "default"])
        resolution = 1.0 if physics == "default" and rng.random() < 0.5 else 0.5
        n = _log(rng, 4e3, 2.5e6)
        cells = n * resolution ** 3  # of water
        side = max(16.0, cells ** (1 / 3) * rng.uniform(1.4, 2.4))
        size = [int(min(160, max(24, side * rng.uniform(0.8, 1.25)))) for _ in range(3)]
        water = rng.choice(["box", "box", "sphere"])
        sub = PHYSICS[physics]["substeps"]
        most = 20 if physics == "bench" else 60
        frames = max(1, int(min(most, 6e7 / n) / sub))
        more = {}
        if water == "box":
            full = (size[0] - 8) * (size[1] - 8) * (size[2] - 8) / resolution ** 3
            f = min(1.0, max(0.05, n / full))
            fx, fz = rng.uniform(f ** 0.5, 1.0), rng.uniform(max(f, f ** 0.5), 1.0)
            more = dict(fx=fx, fy=min(0.9, f / (fx * fz)), fz=fz)
        else:
            r = min(min(size) / 2 - 5.0, max(3.0, (3 * cells / (4 * np.pi)) ** (1 / 3)))
            more = dict(radius=float(r), cy=size[1] / 2.0 - 0.5)
        case = _clip("", physics, size, water, rng.choice(["none", "sphere", "box"]), frames, resolution,
                     rng.choice(["end", "frame"]), **more)
        del case["name"]
        return case
    if kind == "batch":
        return dict(kind="batch", physics=rng.choice(["physical", "bench"]), count=rng.randint(2, 48),
                    frames=rng.randint(2, 5))
    if kind == "learned":
        return dict(kind="learned", steps=rng.randint(2, 10), fx=rng.uniform(0.25, 0.5), fy=rng.uniform(0.1, 0.31),
                    fz=rng.uniform(0.4, 1.0))
    if kind == "train":
        return dict(kind="train", steps=rng.randint(5, 50), batch=64 * int(_log(rng, 16, 1024)), samples=262144)
    if kind == "sdf":
        mesh = rng.choice(["torus", "sphere", "box"])
        sx, sy, sz = (rng.randint(24, 128) for _ in range(3))
        return dict(kind="sdf", sx=sx, sy=sy, sz=sz, mesh=mesh, seg_u=rng.randint(6, 48), seg_v=rng.randint(4, 24),
                    size=min(sx, sy, sz) * rng.uniform(0.1, 0.3))
    if kind == "render":
        return dict(kind="render", n=int(_log(rng, 5e3, 2e6)), width=rng.randint(320, 1920), height=rng.randint(240, 1600),
                    grid=rng.randint(48, 128))
    static = rng.random() < 0.4
    return dict(kind="sort", n=int(_log(rng, 1e3, 1e6 if static else 2e6)), grid=rng.randint(32, 256), static=static)


# ------------------------------------------------------------------ scenes ----
def _jittered(lo, counts, res, keep, gen):
    """Positions (n, 3) float32 on the GPU: one jittered particle per res-sized
    sub-cell of a box at `lo` (x fastest), of the sub-cells keep(centres)."""
    ax = [torch.arange(int(c), device="cuda", dtype=torch.float64) for c in counts]
    zz, yy, xx = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    cell = torch.stack([xx.reshape(-1), yy.reshape(-1), zz.reshape(-1)], 1) * res + torch.as_tensor(lo, device="cuda")
    if keep is not None:
        cell = cell[keep(cell + 0.5 * res)]
    pos = (cell + torch.rand(cell.shape, device="cuda", dtype=torch.float64, generator=gen) * res).float()
    return torch.minimum(pos, (cell + res).float() - 1e-5)


def _box_water(lo, hi, res, gen):
    counts = [int((h - a) / res + 1e-9) for a, h in zip(lo, hi)]
    return _jittered([float(v) for v in lo], counts, res, None, gen)


def _sphere_water(center, radius, res, gen):
    c = torch.tensor(center, dtype=torch.float64, device="cuda")
    m = int(np.ceil(2 * radius / res)) + 1
    return _jittered([float(v) - radius for v in center], (m, m, m), res,
                     lambda p: ((p - c) ** 2).sum(1) < radius * radius, gen)


def _stirred(pos):
    """Initial velocities (n, 3): a gentle eddy, so that the affine matrices
    of a clip's first substeps are not rounding noise around zero."""
    a = pos * (2 * np.pi / 24.0)
    return 0.2 * torch.stack([torch.sin(a[:, 1]), torch.sin(a[:, 2]), torch.sin(a[:, 0])], 1)


def _pinned_state(pos):
    """(26, n) float32 pinned host state in the layout of Engine.init."""
    n = pos.shape[0]
    st = torch.empty((26, n), dtype=torch.float32, pin_memory=True)
    st[0:3].copy_(pos.T.contiguous())
    st[3:6].copy_(_stirred(pos).T.contiguous())
    st[6:24] = 0.0
    st[24:26] = 1.0
    return st.numpy()


def _config(size, physics, resolution=0.5):
    return mpm_b200.Config(size_x=size[0], size_y=size[1], size_z=size[2], resolution=resolution,
                           sdf_resolution=max(size), **PHYSICS[physics])


def _clip_scene(case, seed):
    """(config, positions on the GPU, triangles) of a clip."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    size = (case["sx"], case["sy"], case["sz"])
    res = case["resolution"]
    tris = np.zeros((0, 9), np.float32)
    mid = [s / 2.0 for s in size]
    if case["water"] == "sphere":
        c = [mid[0] + rng.uniform(-0.5, 0.5), case["cy"] + rng.uniform(-0.4, 0.4), mid[2] + rng.uniform(-0.5, 0.5)]
        pos = _sphere_water(c, case["radius"], res, gen)
    elif case["water"] == "box":
        pos = _box_water((4.0, 4.0, 4.0), [4.0 + (s - 8.0) * case[k] for s, k in zip(size, ("fx", "fy", "fz"))], res, gen)
    else:  # three boxes of the 256^3 scene, extents 40-90 cells per axis, about 7M particles
        parts = []
        for ext in ((84.0, 47.0, 61.0), (52.0, 78.5, 66.0), (66.5, 54.0, 90.0)):
            lo = rng.uniform(8.0, 248.0 - np.array(ext))
            parts.append(_box_water(lo, lo + ext, res, gen))
        pos = torch.cat(parts)
    if case["obstacle"] == "torus":
        c = np.array([80.0, 30.0, 64.0]) + rng.uniform(-2.0, 2.0, 3)
        tris = scenes.torus(25.0, 8.0, c, 48, 24)
    elif case["obstacle"] == "sphere":
        tris = scenes.uv_sphere(min(size) / 8.0, [0.75 * size[0], 0.25 * size[1], mid[2]], 24, 12)
    elif case["obstacle"] == "box":
        tris = scenes.box_mesh((size[0] / 6.0, size[1] / 5.0, size[2] / 4.0), [0.7 * size[0], 0.3 * size[1], mid[2]])
    elif case["obstacle"] == "three":
        f = rng.uniform(0.8, 1.2, 3)
        c = rng.uniform(70, 186, (3, 3))
        tris = np.concatenate([scenes.uv_sphere(30 * f[0], c[0]), scenes.torus(50 * f[1], 12 * f[1], c[1]),
                               scenes.box_mesh((60 * f[2], 20 * f[2], 60 * f[2]), c[2])])
    return _config(size, case["physics"], res), pos, tris


def _dam_case(case):
    return _clip("", "physical", (128, 128, 128), "box", "torus", 0, fx=case["fx"], fy=case["fy"], fz=case["fz"])


def _batch_scenes(case, seed):
    """(config, positions, triangles) per scene: grid edges uniform in
    [32, 96], a water sphere of 10k-500k particles, 0-2 obstacles.  The sizes
    are the case's; the seed jitters the particles and shifts the water."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    jit = np.random.default_rng(int(seed))
    rng = np.random.default_rng(1237)
    out = []
    for _ in range(case["count"]):
        size = tuple(int(v) for v in rng.integers(32, 97, size=3))
        ext = float(min(size))
        target = float(np.exp(rng.uniform(np.log(1e4), np.log(5e5))))
        r = float(np.clip((3.0 * target / (32.0 * np.pi)) ** (1.0 / 3.0), 0.2 * ext, 0.4 * ext))
        lo = np.array([4.0 + r] * 3)
        hi = np.maximum(np.array(size, np.float64) - 4.0 - r, lo)
        c = np.clip(rng.uniform(lo, hi) + jit.uniform(-0.5, 0.5, 3), 3.5 + r, np.array(size) - 3.5 - r)
        tris = []
        for _k in range(int(rng.integers(0, 3))):
            oc = rng.uniform(0.2, 0.8, size=3) * np.array(size)
            s = float(rng.uniform(0.1, 0.2) * ext)
            tris.append(scenes.torus(s, s / 3.0, tuple(oc), 24, 12) if rng.random() < 0.5
                        else scenes.box_mesh((s, s / 2.0, s), tuple(oc)))
        out.append((_config(size, case["physics"]), _sphere_water([float(v) for v in c], r, 0.5, gen),
                    np.concatenate(tris) if tris else np.zeros((0, 9), np.float32)))
    return out


def _mesh(case, seed):
    rng = np.random.default_rng(int(seed))
    size = np.array([case["sx"], case["sy"], case["sz"]], np.float64)
    c = size / 2 + rng.uniform(-0.08, 0.08, 3) * size
    s = case["size"] * rng.uniform(0.95, 1.05)
    if case["mesh"] == "torus":
        return scenes.torus(s, s * 0.32, c, case["seg_u"], case["seg_v"])
    if case["mesh"] == "sphere":
        return scenes.uv_sphere(s, c, case["seg_u"], case["seg_v"])
    return scenes.box_mesh((2 * s, s, 1.5 * s), c)


def _weights(physical=True):
    return learned.load_params(learned.PHYSICAL_PARAMS if physical else learned.DEFAULT_PARAMS)[0]


def _training_rows(case, seed):
    """Features with the spread the collection probe records (affine matrix,
    velocity, density, folded distance) and targets that depend on them."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n = case["samples"]
    z = torch.randn((n, 16), device="cuda", generator=gen)
    f = z * torch.tensor([0.15] * 9 + [0.8, 1.2, 0.6] + [1.5] + [0.4] * 3, device="cuda")
    f[:, 12] = f[:, 12].abs()
    t = 0.1 * torch.tanh(f[:, 9:12]) + 0.2 * f[:, [0, 4, 8]] + 0.05 * torch.randn((n, 3), device="cuda", generator=gen)
    return f.cpu().numpy(), t.cpu().numpy()


def _cloud(case, seed):
    """Positions of a dam-break-like block on its way (original order: x
    fastest, each particle about a cell from where it was seeded), (n, 3)."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n, g = case["n"], case["grid"]
    span = g - 8.0
    res = min(0.5, (0.4667 * 0.3084 * span ** 3 / n) ** (1 / 3))
    nx, nz = int(0.4667 * span / res), int(span / res)
    ny = -(-n // (nx * nz))
    pos = _jittered([4.0, 4.0, 4.0], (nx, ny, nz), res, None, gen)[:n]
    return (pos + torch.randn(pos.shape, device="cuda", generator=gen)).clamp(3.0, g - 3.0).contiguous()


# ------------------------------------------------------------------ prepare ----
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "clip":
        cfg, pos, tris = _clip_scene(case, seed)
        s["engine"] = e = mpm_b200.Engine(cfg)
        s["state"] = _pinned_state(pos)
        s["out"] = torch.empty((26, pos.shape[0]), dtype=torch.float32, pin_memory=True).numpy()
        s["frame"] = torch.empty((pos.shape[0], 3), dtype=torch.float32, pin_memory=True).numpy()
        if len(tris):
            e.init_sdf(tris)
    elif kind == "batch":
        made = _batch_scenes(case, seed)
        s["engine"] = e = mpm_b200.Batch([m[0] for m in made])
        s["states"] = [_pinned_state(m[1]) for m in made]
        s["outs"] = [torch.empty((26, m[1].shape[0]), dtype=torch.float32, pin_memory=True).numpy() for m in made]
        for k, m in enumerate(made):
            if len(m[2]):
                e.init_scene_sdf(k, m[2])
    elif kind == "learned":
        cfg, pos, tris = _clip_scene(_dam_case(case), seed)
        s["engine"] = e = mpm_b200.Engine(cfg)
        s["state"] = _pinned_state(pos)
        s["out"] = torch.empty((26, pos.shape[0]), dtype=torch.float32, pin_memory=True).numpy()
        e.init_sdf(tris)
        e.set_corrector(_weights(), ratio=4, max_density_change=-1.0)
    elif kind == "train":
        f, t = _training_rows(case, seed)
        s["corrector"] = c = mpm_b200.Corrector(case["samples"])
        c.add_data(f, t)
        c.init(seed=int(seed))
    elif kind == "sdf":
        cfg = _config((case["sx"], case["sy"], case["sz"]), "bench")
        s["engine"] = mpm_b200.Engine(cfg)
        s["tris"] = _mesh(case, seed)
    elif kind == "render":
        s["pos"] = _cloud(case, seed)
        g = case["grid"]
        s["renderer"] = mpm_b200.Renderer((g, g, g), case["width"], case["height"])
    else:
        pos = _cloud(case, seed)
        s["planes"] = pos.T.contiguous()
        s["keys"] = torch.empty(pos.shape[0], dtype=torch.int32, device="cuda")
        s["perm"] = torch.empty_like(s["keys"])
    return s


# ---------------------------------------------------------------------- run ----
def _fields(st):
    return {"position": st[0:3], "velocity": st[3:6], "affine": st[6:15], "deformation": st[15:24],
            "volume_mass": st[24:26]}


def _read_state(engine, out):
    engine._check(mpm_b200.lib.mpm_get_state(engine._h, out.ctypes.data))
    return _fields(out)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "clip":
        e = s["engine"]
        e.init(s["state"])
        for _ in range(case["frames"]):
            e.step(e.cfg.substeps)
            if case["read"] == "frame":
                e.get_positions(s["frame"])
        return _read_state(e, s["out"])
    if kind == "batch":
        e = s["engine"]
        e.init_all(s["states"])
        for _ in range(case["frames"]):
            e.step(e.cfg.substeps)
        for k, out in enumerate(s["outs"]):
            e._check(mpm_b200.lib.mpm_scene_get_state(e._h, k, out.ctypes.data))
        return s["outs"]
    if kind == "learned":
        e = s["engine"]
        e.init(s["state"])
        e.step_learned(case["steps"])
        return _read_state(e, s["out"])
    if kind == "train":
        c = s["corrector"]
        loss = c.train(case["steps"], batch=case["batch"], lr=1e-3, seed=3)
        return {"loss": loss, "params": c.get_params()}
    if kind == "sdf":
        s["engine"].init_sdf(s["tris"])
        return s["engine"].get_sdf()
    if kind == "render":
        r, p = s["renderer"], s["pos"]
        r.render_device(p.data_ptr(), p.shape[0], torch.cuda.current_stream().cuda_stream)
        rgb, rgb8 = r.image()
        return {"rgb": rgb, "rgb8": rgb8}
    p = s["planes"]
    sort = mpm_b200.sort_particles_device_static if case["static"] else mpm_b200.sort_particles_device
    sort(p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), p.shape[1], s["keys"].data_ptr(), s["perm"].data_ptr(),
         torch.cuda.current_stream().cuda_stream)
    return {"keys": s["keys"], "perm": s["perm"]}


# --------------------------------------------------------------------- work ----
# Per particle and substep: the 96-byte state read and written once and its
# position, F read again by the gather (48 bytes); about 1000 operations of
# scatter and gather.  The upload is 21 planes, the read-back 26.
def _clip_work(n, substeps):
    return {"bytes": n * (substeps * 240.0 + 4.0 * 47), "flops": n * substeps * 1000.0}


def _box_count(size, f, res):
    return float(np.prod([int((s - 8.0) * k / res) for s, k in zip(size, f)]))


def _count(case):
    res = case["resolution"]
    if case["water"] == "sphere":
        return 4.0 / 3.0 * np.pi * (case["radius"] / res) ** 3
    if case["water"] == "box":
        return _box_count((case["sx"], case["sy"], case["sz"]), (case["fx"], case["fy"], case["fz"]), res)
    return (84.0 * 47.0 * 61.0 + 52.0 * 78.5 * 66.0 + 66.5 * 54.0 * 90.0) / res ** 3


def work(case):
    kind = case["kind"]
    if kind == "clip":
        return _clip_work(_count(case), case["frames"] * PHYSICS[case["physics"]]["substeps"])
    if kind == "batch":
        rng, n = np.random.default_rng(1237), 0.0
        for _ in range(case["count"]):  # the scenes' spheres, drawn as in _batch_scenes
            size = rng.integers(32, 97, size=3)
            ext = float(min(size))
            r = float(np.clip((3.0 * np.exp(rng.uniform(np.log(1e4), np.log(5e5))) / (32.0 * np.pi)) ** (1.0 / 3.0),
                              0.2 * ext, 0.4 * ext))
            rng.uniform(0, 1, 3)
            for _k in range(int(rng.integers(0, 3))):
                rng.uniform(0, 1, 5)
            n += 4.0 / 3.0 * np.pi * (r / 0.5) ** 3
        return _clip_work(n, case["frames"] * PHYSICS[case["physics"]]["substeps"])
    if kind == "learned":
        n = _box_count((128,) * 3, (case["fx"], case["fy"], case["fz"]), 0.5)
        w = _clip_work(n, case["steps"])
        return {"bytes": w["bytes"], "flops": w["flops"] + n * case["steps"] * 2.0 * (16 * 64 + 64 * 64 + 64 * 3)}
    if kind == "train":
        rows = float(case["steps"]) * case["batch"]
        return {"bytes": rows * 76.0, "flops": rows * 6.0 * (16 * 64 + 64 * 64 + 64 * 3)}
    if kind == "sdf":
        # a nearest triangle and a sign per node: about 200 operations each
        g = float(case["sx"] * case["sy"] * case["sz"])
        return {"bytes": 4.0 * g, "flops": 400.0 * g}
    if kind == "render":
        px = float(case["width"] * case["height"])
        return {"bytes": 12.0 * case["n"] + 15.0 * px, "flops": px * 2 * 21 * 10.0 + 50.0 * case["n"]}
    return {"bytes": 20.0 * case["n"], "flops": 20.0 * case["n"]}


# -------------------------------------------------------------------- exact ----
def _distance(nodes, tris):
    """Signed distance of points (m, 3) to triangles (t, 9), float64."""
    A, B, C = tris[:, 0:3], tris[:, 3:6], tris[:, 6:9]
    nrm = torch.linalg.cross(B - A, C - A)
    nn = (nrm * nrm).sum(1)
    out = torch.empty(nodes.shape[0], dtype=torch.float64, device=nodes.device)
    step = max(1, int(1.5e7 // tris.shape[0]))
    for i in range(0, nodes.shape[0], step):
        p = nodes[i:i + step, None, :]
        a, b, c = A[None] - p, B[None] - p, C[None] - p
        la, lb, lc = a.norm(dim=2), b.norm(dim=2), c.norm(dim=2)
        det = (a * torch.linalg.cross(b, c)).sum(2)
        div = la * lb * lc + (a * b).sum(2) * lc + (a * c).sum(2) * lb + (b * c).sum(2) * la
        wn = (2.0 * torch.atan2(det, div)).sum(1) / (4 * 3.1415)
        d2 = None
        inside = None
        for u, v in ((a, b), (b, c), (c, a)):
            e = v - u
            t = (-(u * e).sum(2) / (e * e).sum(2).clamp_min(1e-300)).clamp(0, 1)
            q = u + t[..., None] * e
            s = (q * q).sum(2)
            d2 = s if d2 is None else torch.minimum(d2, s)
            side = (torch.linalg.cross(e, -u) * nrm[None]).sum(2) >= 0
            inside = side if inside is None else inside & side
        h = (a * nrm[None]).sum(2) ** 2 / nn[None].clamp_min(1e-300)
        d2 = torch.where(inside & (nn[None] > 0), torch.minimum(h, d2), d2)
        out[i:i + step] = torch.where(wn > 0.5, -1.0, 1.0) * d2.min(1).values.sqrt()
    return out


def _grid_nodes(lo, hi):
    ax = [torch.arange(int(a), int(b), device="cuda", dtype=torch.float64) for a, b in zip(lo, hi)]
    zz, yy, xx = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack([xx.reshape(-1), yy.reshape(-1), zz.reshape(-1)], 1)


def _near_sdf(size, tris):
    """The distance field near the obstacles; far nodes hold +1e3 (no particle
    or node there is affected by its value)."""
    sx, sy, sz = size
    sdf = torch.full((sx * sy * sz,), 1e3, dtype=torch.float64, device="cuda")
    if not len(tris):
        return sdf
    t = torch.as_tensor(np.asarray(tris, np.float64), device="cuda")
    v = t.reshape(-1, 3, 3)
    near = torch.zeros((sz, sy, sx), dtype=torch.bool, device="cuda")
    lo, hi = (v.min(1).values - 8).floor().long(), (v.max(1).values + 9).ceil().long()
    for a, b in zip(lo.tolist(), hi.tolist()):
        a, b = [max(0, x) for x in a], [max(0, x) for x in b]
        near[a[2]:b[2], a[1]:b[1], a[0]:b[0]] = True
    # interiors: the box of all triangles around what is marked
    l, h = lo.min(0).values.clamp_min(0).tolist(), hi.max(0).values.clamp_min(0).tolist()
    vol = (h[0] - l[0]) * (h[1] - l[1]) * (h[2] - l[2])
    if vol <= 4e6:
        near[l[2]:h[2], l[1]:h[1], l[0]:h[0]] = True
    idx = near.reshape(-1).nonzero()[:, 0]
    nodes = torch.stack([idx % sx, (idx // sx) % sy, idx // (sx * sy)], 1).double()
    sdf[idx] = _distance(nodes, t)
    return sdf


class _Exact:
    """One scene's substeps in float64 (the MLS-MPM step of the engine)."""

    def __init__(self, cfg, pos, tris):
        self.c, self.n = cfg, pos.shape[0]
        f32 = lambda v: float(np.float32(v))
        self.dt, self.g, self.gamma, self.k = f32(cfg.dt), f32(cfg.gravity), f32(cfg.gamma), f32(cfg.compression)
        self.vol = f32(cfg.resolution) ** 3
        self.size = torch.tensor([cfg.size_x, cfg.size_y, cfg.size_z], device="cuda")
        self.x = pos.double()
        self.v = _stirred(pos).double()
        self.C = torch.zeros((self.n, 3, 3), dtype=torch.float64, device="cuda")
        self.F = torch.eye(3, dtype=torch.float64, device="cuda").expand(self.n, 3, 3).clone()
        self.sdf = _near_sdf((cfg.size_x, cfg.size_y, cfg.size_z), tris)
        sx, sy, sz = cfg.size_x, cfg.size_y, cfg.size_z
        self.G = sx * sy * sz
        i = torch.arange(self.G, device="cuda")
        self.node = [i % sx, (i // sx) % sy, i // (sx * sy)]
        self.neg = (self.sdf < 0).nonzero()[:, 0]

    def index(self, q):
        return (q[:, 2] * self.c.size_y + q[:, 1]) * self.c.size_x + q[:, 0]

    def stencil(self, x):
        base = (x - 0.5).trunc().long()
        f = x - base
        w = []
        for a in range(3):
            d = (f - a).abs()
            w.append(torch.where(d < 0.5, 0.75 - d * d, torch.where(d < 1.5, 0.5 * (1.5 - d) ** 2, 0.0 * d)))
        for a in range(3):
            for b in range(3):
                for c in range(3):
                    o = torch.tensor([a, b, c], device="cuda")
                    q = base + o
                    ok = ((q >= 0) & (q < self.size)).all(1)
                    wt = torch.where(ok, w[a][:, 0] * w[b][:, 1] * w[c][:, 2], 0.0)
                    yield self.index(torch.minimum(q.clamp_min(0), self.size - 1)), wt, q.double() - x

    def grid(self, dt):
        J = torch.linalg.det(self.F).clamp(0.9, 1.1)
        pressure = (self.k * (J ** self.gamma - 1)).clamp_min(0)
        A = self.C + (4 * dt * self.vol * J * pressure)[:, None, None] * torch.eye(3, dtype=torch.float64, device="cuda")
        grid = torch.zeros((self.G, 4), dtype=torch.float64, device="cuda")
        for idx, w, d in self.stencil(self.x):
            mom = self.v + (A @ d[:, :, None])[:, :, 0]
            grid.index_add_(0, idx, torch.cat([w[:, None], w[:, None] * mom], 1))
        m = grid[:, :1]
        vel = torch.where(m > 1e-9, grid[:, 1:] / m.clamp_min(1e-300), 0.0)
        vel[:, 1] -= torch.where(m[:, 0] > 1e-9, self.g * dt, 0.0)
        if len(self.neg):
            p = torch.stack([self.node[k][self.neg] for k in range(3)], 1)
            nrm = torch.empty((len(self.neg), 3), dtype=torch.float64, device="cuda")
            for k in range(3):
                o = torch.zeros(3, dtype=torch.long, device="cuda")
                o[k] = 1
                hi, lo = torch.minimum(p + o, self.size - 1), (p - o).clamp_min(0)
                nrm[:, k] = self.sdf[self.index(hi)] - self.sdf[self.index(lo)]
            nrm /= nrm.norm(dim=1, keepdim=True) + 1e-9
            vn = vel[self.neg]
            vdn = (vn * nrm).sum(1, keepdim=True).clamp_max(0)
            vel[self.neg] = vn - nrm * vdn
        pad = self.c.padding
        for k in range(3):
            s = int(self.size[k])
            vel[:, k] = torch.where((self.node[k] < pad) & (vel[:, k] < 0), 0.0, vel[:, k])
            vel[:, k] = torch.where((self.node[k] > s - 1 - pad) & (vel[:, k] > 0), 0.0, vel[:, k])
        return m[:, 0], torch.where(m > 1e-9, vel, 0.0)

    def sample(self, q):
        i = q.floor()
        t = q - i
        i = i.long()
        c = lambda o: torch.minimum((i + torch.tensor(o, device="cuda")).clamp_min(0), self.size - 1)
        at = lambda o: self.sdf[self.index(c(o))]
        mix = lambda a, b, s: a * (1 - s) + b * s
        x = [mix(at((0, j, k)), at((1, j, k)), t[:, 0]) for k in (0, 1) for j in (0, 1)]
        return mix(mix(x[0], x[1], t[:, 1]), mix(x[2], x[3], t[:, 1]), t[:, 2])

    def normal(self, q):
        e = 0.1 * torch.eye(3, dtype=torch.float64, device="cuda")
        n = torch.stack([self.sample(q + e[k]) - self.sample(q - e[k]) for k in range(3)], 1)
        return n / (n.norm(dim=1, keepdim=True) + 1e-6)

    def step(self, ratio=1, mlp=None):
        dt = self.dt * ratio
        mass, vel = self.grid(dt)
        v = torch.zeros_like(self.v)
        C = torch.zeros_like(self.C)
        rho = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        for idx, w, d in self.stencil(self.x):
            g = w[:, None] * vel[idx]
            v += g
            C += 4 * g[:, :, None] * d[:, None, :]
            if mlp is not None:
                rho += w * mass[idx]
        if mlp is not None:
            phi = self.sample(self.x)
            near = phi.abs() < 4
            fold = torch.zeros_like(v)
            fold[near] = self.normal(self.x[near]) * (phi[near] * (1 - phi[near].abs() / 4))[:, None]
            v = v + mlp(torch.cat([C.reshape(-1, 9), v, (rho * self.vol - 1)[:, None], fold], 1))
        F = (torch.eye(3, dtype=torch.float64, device="cuda") + dt * C) @ self.F
        J = torch.linalg.det(F)
        scale = torch.where(J < 0.3, (0.3 / J) ** (1.0 / 3.0), 1.0)
        self.F = F * scale[:, None, None]
        adv = v if ratio == 1 else self.v + (ratio + 1) / (2.0 * ratio) * (v - self.v)
        x = self.x + adv * dt
        d = self.sample(x)
        hit = (d < 0).nonzero()[:, 0]
        if len(hit):
            nrm = self.normal(x[hit])
            x[hit] -= nrm * d[hit][:, None]
            v[hit] -= nrm * (v[hit] * nrm).sum(1, keepdim=True).clamp_max(0)
        self.x, self.v, self.C = x, v, C

    def state(self):
        st = torch.empty((26, self.n), dtype=torch.float64, device="cuda")
        st[0:3], st[3:6] = self.x.T, self.v.T
        st[6:15], st[15:24] = self.C.reshape(-1, 9).T, self.F.reshape(-1, 9).T
        st[24], st[25] = self.vol, 1.0
        return st


def _mlp64(w):
    w = torch.as_tensor(np.asarray(w, np.float64), device="cuda")
    sizes = (16, 16, 3, 64 * 16, 64, 64 * 64, 64, 3 * 64, 3)
    mean, inv, scale, W1, b1, W2, b2, W3, b3 = torch.split(w, sizes)
    gelu = lambda h: torch.nn.functional.gelu(h, approximate="tanh")

    def net(x):
        h = gelu(((x - mean) * inv) @ W1.reshape(64, 16).T + b1)
        h = gelu(h @ W2.reshape(64, 64).T + b2)
        return (h @ W3.reshape(3, 64).T + b3) * scale
    return net


def exact(case, seed):
    kind = case["kind"]
    if kind == "clip":
        cfg, pos, tris = _clip_scene(case, seed)
        s = _Exact(cfg, pos, tris)
        for _ in range(case["frames"] * cfg.substeps):
            s.step()
        return _fields(s.state())
    if kind == "batch":
        out = []
        for cfg, pos, tris in _batch_scenes(case, seed):
            s = _Exact(cfg, pos, tris)
            for _ in range(case["frames"] * cfg.substeps):
                s.step()
            out.append(s.state().cpu())
        return out
    if kind == "learned":
        cfg, pos, tris = _clip_scene(_dam_case(case), seed)
        s = _Exact(cfg, pos, tris)
        net = _mlp64(_weights())
        for _ in range(case["steps"]):
            s.step(4, net)
        return _fields(s.state())
    if kind == "sdf":
        tris = torch.as_tensor(_mesh(case, seed).astype(np.float64), device="cuda")
        return _distance(_grid_nodes((0, 0, 0), (case["sx"], case["sy"], case["sz"])), tris)
    # train: its samples are drawn by the library's own generator; render: the
    # image is defined by its float32 roundings (which pixels a sprite covers);
    # sort: whole numbers.
    return None
