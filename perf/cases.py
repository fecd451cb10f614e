"""Performance cases: what a user of the renderer has it do, at the sizes it is used at.

Every case goes through the Python mirror of the C ABI (``voxeltoy_gb300``):
a viewer's progressive passes, finished frames of the benchmark's scene
families, many jobs in one call, requests to the render server, meshes
voxelized and shown, volumes loaded and environment maps built.  Host arrays
in, host arrays out, as the C ABI takes and returns them.

The images have no 64-bit values here: a path traced in 64 bits meets another
voxel than the 32-bit one wherever a ray grazes an edge, and a plain 64-bit
trace of these frames takes minutes.  The environment's CDFs have them.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from voxeltoy_gb300 import Context, Env, Job, Scene, Server
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

SPHERES, FBM, SHELL = "spheres", "fbm", "shell"

_context = None


def context() -> Context:
    """One context for the process, as a program that renders keeps one."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


# ------------------------------------------------------------------- cases
def _frame(name, scene, res, size, spp, bounces, rr=-1, env=(0, 0), lens=False, noise=False, reference=False):
    c = {"kind": "frame", "scene": scene, "rx": res[0], "ry": res[1], "rz": res[2], "w": size[0], "h": size[1],
         "spp": spp, "bounces": bounces, "rr": rr, "env_w": env[0], "env_h": env[1], "lens": lens, "noise": noise,
         "reference": reference}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one progressive pass of a small preview while the camera moves: launches and latency
        _frame("pass_preview", SPHERES, (64, 64, 64), (160, 120), 1, 4),
        # one progressive pass of a viewer's window, with every shading feature on
        _frame("pass_window", FBM, (128, 128, 128), (512, 512), 1, 8, rr=3, env=(512, 256), lens=True),
        # the smallest benchmark frame: 64^3 spheres, 256^2, 16 samples, white sky
        _frame("frame_spheres", SPHERES, (64, 64, 64), (256, 256), 16, 4),
        # the headline frame: 256^3, 1024^2, 256 samples, sky and sun, thin lens, roulette
        _frame("frame_full", FBM, (256, 256, 256), (1024, 1024), 256, 8, rr=3, env=(1024, 512), lens=True),
        # a volume and an image with no round size, the reference's quirks and its noise-table stream
        _frame("frame_ragged", FBM, (203, 117, 89), (641, 479), 7, 5, noise=True, reference=True),
        # the largest volume: a voxelized closed surface, nearly empty space
        _frame("frame_shell", SHELL, (1024, 1024, 1024), (1024, 1024), 16, 8, env=(1024, 512)),
        # uneven scenes and images in one call
        {"name": "batch_mixed", "kind": "batch", "jobs": 24, "edge_min": 32, "edge_max": 224, "spp": 16, "bounces": 4},
        # requests of several sizes and sample targets that reach the server together
        {"name": "serve_mixed", "kind": "serve", "jobs": 12, "edge_min": 64, "edge_max": 192, "spp": 64, "bounces": 4},
        # a large mesh voxelized conservatively and looked at: the first edit-mode image of it
        {"name": "mesh_view", "kind": "mesh", "rows": 572, "rx": 1024, "ry": 1024, "rz": 1024, "fat": True,
         "w": 512, "h": 512, "voxels": False},
        # a small mesh turned into a thin voxel grid that is read back
        {"name": "mesh_grid", "kind": "mesh", "rows": 70, "rx": 96, "ry": 128, "rz": 80, "fat": False,
         "w": 0, "h": 0, "voxels": True},
        # a dense volume loaded, its emissive voxels found and pruned
        {"name": "load_volume", "kind": "load", "rx": 256, "ry": 256, "rz": 256},
        # an HDR environment map made ready for sampling
        {"name": "env_build", "kind": "env", "env_w": 1024, "env_h": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "shell", "batch", "serve", "mesh", "load", "env"])
    if kind == "frame":
        scene = rng.choice([SPHERES, FBM])
        res = tuple(_log(rng, 24, 288) for _ in range(3))
        size = (_log(rng, 96, 1100), _log(rng, 64, 900))
        spp = _log(rng, 1, 64)
        env = rng.choice([(0, 0), (_log(rng, 64, 1024), _log(rng, 32, 512))])
        return _frame(None, scene, res, size, spp, rng.randint(1, 9), rr=rng.choice([-1, 2, 3]), env=env,
                      lens=rng.random() < 0.5, noise=rng.random() < 0.25, reference=rng.random() < 0.25)
    if kind == "shell":
        edge = _log(rng, 200, 1024)
        size = (_log(rng, 160, 1100), _log(rng, 120, 1000))
        return _frame(None, SHELL, (edge, edge, edge), size, _log(rng, 1, 24), rng.randint(2, 8),
                      env=rng.choice([(0, 0), (512, 256)]))
    if kind == "batch":
        return {"kind": "batch", "jobs": _log(rng, 2, 40), "edge_min": 32, "edge_max": _log(rng, 64, 256),
                "spp": _log(rng, 2, 32), "bounces": rng.randint(2, 6)}
    if kind == "serve":
        return {"kind": "serve", "jobs": _log(rng, 2, 16), "edge_min": 64, "edge_max": _log(rng, 96, 224),
                "spp": _log(rng, 16, 128), "bounces": rng.randint(2, 6)}
    if kind == "mesh":
        if rng.random() < 0.5:
            return {"kind": "mesh", "rows": _log(rng, 24, 572), "rx": _log(rng, 64, 1024), "ry": _log(rng, 64, 1024),
                    "rz": _log(rng, 64, 1024), "fat": rng.random() < 0.7, "w": _log(rng, 160, 1024),
                    "h": _log(rng, 120, 768), "voxels": False}
        return {"kind": "mesh", "rows": _log(rng, 16, 200), "rx": _log(rng, 24, 256), "ry": _log(rng, 24, 256),
                "rz": _log(rng, 24, 256), "fat": rng.random() < 0.5, "w": 0, "h": 0, "voxels": True}
    if kind == "load":
        return {"kind": "load", "rx": _log(rng, 24, 320), "ry": _log(rng, 24, 320), "rz": _log(rng, 24, 320)}
    return {"kind": "env", "env_w": _log(rng, 64, 2048), "env_h": _log(rng, 32, 1024)}


# ------------------------------------------------------------------ inputs
def _spheres(res, seed):
    """A union of spheres over a ground slab (uint8 [z, y, x], palette entry 1)."""
    rng = random.Random(seed)
    rx, ry, rz = res
    g = torch.zeros((rz, ry, rx), dtype=torch.uint8, device="cuda")
    g[:, :max(1, ry // 16), :] = 1
    small = min(res)
    zz = torch.arange(rz, device="cuda", dtype=torch.float32)[:, None, None] + 0.5
    yy = torch.arange(ry, device="cuda", dtype=torch.float32)[None, :, None] + 0.5
    xx = torch.arange(rx, device="cuda", dtype=torch.float32)[None, None, :] + 0.5
    for _ in range(rng.randint(8, 14)):
        cx, cy, cz = rng.uniform(0, rx), rng.uniform(0, ry), rng.uniform(0, rz)
        r = rng.uniform(0.09, 0.25) * small
        g |= ((xx - cx) ** 2 + (yy - cy) ** 2 + (zz - cz) ** 2 <= r * r).to(torch.uint8)
    return g.cpu().numpy()


def _fbm(res, seed, octaves=3, base_cells=8, occupancy=0.35):
    """Three octaves of value noise thresholded to the given occupancy, random
    palette entries 1..16 and 2% of the occupied voxels emissive (entry 17)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    shape = (res[2], res[1], res[0])
    field = torch.zeros(shape, dtype=torch.float32, device="cuda")
    for o in range(octaves):
        cells = base_cells * 2 ** o
        a = torch.rand((cells + 1,) * 3, generator=gen, device="cuda")
        for axis in (2, 1, 0):
            n = shape[axis]
            t = (torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * (cells / n)
            i0 = t.floor().long().clamp(max=cells - 1)
            f = t - i0
            view = [1, 1, 1]
            view[axis] = n
            s = (f * f * (3.0 - 2.0 * f)).view(view)
            a = a.index_select(axis, i0) * (1.0 - s) + a.index_select(axis, i0 + 1) * s
        field += 0.5 ** o * a
    flat = field.flatten()
    level = flat.sort().values[int((1.0 - occupancy) * flat.numel())]
    solid = field >= level
    g = torch.randint(1, 17, shape, generator=gen, device="cuda", dtype=torch.uint8)
    lit = torch.rand(shape, generator=gen, device="cuda") < 0.02
    g[lit] = 17
    g[~solid] = 0
    return g.cpu().numpy()


def _mesh(rows, seed):
    """A closed sphere of 4 rows^2 triangles or so, its radius moved by smooth waves of four octaves."""
    rng = np.random.default_rng(seed)
    cols = 2 * rows
    theta = np.linspace(0.0, math.pi, rows + 1)[:, None]
    phi = np.arange(cols)[None, :] * (2.0 * math.pi / cols)
    p = np.stack([np.sin(theta) * np.cos(phi), np.cos(theta) * np.ones_like(phi), np.sin(theta) * np.sin(phi)], -1)
    move = np.zeros(p.shape[:2])
    for o in range(4):
        for _ in range(3):
            k = rng.normal(0.0, 2.0 ** (o + 1), 3)
            move += 0.5 ** o * np.sin(p @ k + rng.uniform(0.0, 2.0 * math.pi))
    v = (p * (1.0 + 0.15 * move / 6.0)[..., None]).reshape(-1, 3).astype(np.float32)
    i, j = np.meshgrid(np.arange(rows), np.arange(cols), indexing="ij")
    j1 = (j + 1) % cols
    a, b, c, d = i * cols + j, (i + 1) * cols + j, (i + 1) * cols + j1, i * cols + j1
    lower = np.stack([a, b, c], -1)[:-1].reshape(-1, 3)     # the last row's lower triangles have no area
    upper = np.stack([a, c, d], -1)[1:].reshape(-1, 3)      # nor have the first row's upper ones
    return v, np.concatenate([lower, upper]).astype(np.uint32)


def _sky(w, h, seed):
    rng = random.Random(seed)
    return S.sky_sun_env(w, h, sun_elevation_deg=rng.uniform(20.0, 70.0), sun_azimuth_deg=rng.uniform(-180.0, 180.0))


def _camera(seed, lens=False):
    rng = random.Random(seed + 1)
    return S.orbit_camera(distance=rng.uniform(1500.0, 2200.0), theta_deg=rng.uniform(100.0, 140.0),
                          phi_deg=rng.uniform(0.0, 360.0),
                          lens=L.VT_LENS_THIN_LENS if lens else L.VT_LENS_PINHOLE, aperture=20.0 if lens else 0.0)


def _image(w, h):
    """The pinned host buffer that a program reads its frames into."""
    return torch.empty((h, w, 4), dtype=torch.float32, pin_memory=True).numpy()


def _scene(ctx, scene, res, seed):
    if scene == SHELL:
        v, i = _mesh(400, seed)
        return Scene.voxelize(ctx, v, i, res, L.VT_VOXELIZE_FAT)
    if scene == SPHERES:
        return Scene.dense(ctx, _spheres(res, seed), [S.lambert(0.7)])
    return Scene.dense(ctx, _fbm(res, seed), S.config2_palette(seed),
                       flags=L.VT_SCENE_AUTO_EMISSIVE | L.VT_SCENE_PRUNE_EMISSIVE)


class State:
    """What the program holds; handles close in the order they were added."""

    def __init__(self, case):
        self.case = case
        self.held = []

    def hold(self, x):
        self.held.append(x)
        return x

    def __del__(self):
        for x in self.held:
            x.close()


def _several(st, case, seed):
    """Scenes, cameras, sizes and sample targets of a batch or a request stream; the sizes are the case's own."""
    rng = random.Random(case["jobs"] * 4096 + case["edge_max"])
    ctx = context()
    out = []
    for k in range(case["jobs"]):
        edge = _log(rng, case["edge_min"], case["edge_max"])
        w, h = rng.choice([128, 192, 256, 384, 512]), rng.choice([128, 192, 256, 384, 512])
        scene = Scene.dense(ctx, _spheres((edge, edge, edge), seed * 1000 + k), [S.lambert(0.7)])
        out.append((scene, _camera(seed * 1000 + k), S.physical_settings(case["bounces"], seed=seed + k), w, h,
                    max(1, _log(rng, max(1, case["spp"] // 8), case["spp"]))))
    return out


def prepare(case, seed):
    ctx = context()
    st = State(case)
    kind = case["kind"]
    if kind == "frame":
        res = (case["rx"], case["ry"], case["rz"])
        scene = _scene(ctx, case["scene"], res, seed)
        env = Env(ctx, _sky(case["env_w"], case["env_h"], seed)) if case["env_w"] else None
        s = S.physical_settings(case["bounces"], case["rr"], seed=seed, top=(0.9, 1.0, 1.1), bottom=(0.5, 0.5, 0.5))
        if case["reference"]:
            # unguarded samples left out: they turn pixels into NaN for good
            s.quirks = L.VT_QUIRKS_REFERENCE & ~L.VT_QUIRK_UNGUARDED_SAMPLES
        if case["noise"]:
            s.rng_mode = L.VT_RNG_NOISE_TABLE
        st.camera = _camera(seed, case["lens"])
        st.job = st.hold(Job(ctx, scene, env, st.camera, s, case["w"], case["h"]))
        st.hold(scene)
        if env:
            st.hold(env)
        st.image = _image(case["w"], case["h"])
    elif kind == "batch":
        made = _several(st, case, seed)
        st.jobs = [st.hold(Job(ctx, sc, None, cam, s, w, h)) for sc, cam, s, w, h, _spp in made]
        for m in made:
            st.hold(m[0])
        st.images = [_image(j.width, j.height) for j in st.jobs]
    elif kind == "serve":
        st.requests = _several(st, case, seed)
        st.server = st.hold(Server(ctx))
        for m in st.requests:
            st.hold(m[0])
    elif kind == "mesh":
        st.vertices, st.indices = _mesh(case["rows"], seed)
        if not case["voxels"]:
            st.image = _image(case["w"], case["h"])
            st.camera = _camera(seed)
            st.settings = S.physical_settings(4, seed=seed)
    elif kind == "load":
        st.voxels = _fbm((case["rx"], case["ry"], case["rz"]), seed)
        st.palette = S.config2_palette(seed)
        # room for every emissive voxel (0.7% of the volume's), -1 after the last
        st.emissive = np.full(64 + st.voxels.size // 80, -1, np.int32)
    else:
        st.sky = _sky(case["env_w"], case["env_h"], seed)
    return st


# --------------------------------------------------------------------- run
def run(st):
    case, ctx = st.case, context()
    kind = case["kind"]
    if kind == "frame":           # the camera is set (which restarts the image), passes are added, the image is read
        st.job.set_camera(st.camera)
        st.job.render(case["spp"])
        return st.job.readback(out=st.image)
    if kind == "batch":
        for j in st.jobs:
            j.reset()
        ctx.render_batch(st.jobs, case["spp"])
        return [j.readback(out=o) for j, o in zip(st.jobs, st.images)]
    if kind == "serve":
        tickets = [st.server.submit(sc, None, cam, s, w, h, spp) for sc, cam, s, w, h, spp in st.requests]
        out = []
        for t, (_sc, _cam, _s, w, h, _spp) in zip(tickets, st.requests):
            if st.server.wait(t) != L.VT_OK:
                raise RuntimeError("request failed")
            out.append(st.server.result(t, w, h)[0])
        return out
    if kind == "mesh":
        scene = Scene.voxelize(ctx, st.vertices, st.indices, (case["rx"], case["ry"], case["rz"]),
                               L.VT_VOXELIZE_FAT if case["fat"] else L.VT_VOXELIZE_THIN)
        try:
            if case["voxels"]:
                return scene.voxels()
            job = Job(ctx, scene, None, st.camera, st.settings, case["w"], case["h"])
            try:
                job.set_integrator(L.VT_INTEGRATOR_EDIT_MODE)
                job.render(1)
                return job.readback(out=st.image)
            finally:
                job.close()
        finally:
            scene.close()
    if kind == "load":
        scene = Scene.dense(ctx, st.voxels, st.palette,
                            flags=L.VT_SCENE_AUTO_EMISSIVE | L.VT_SCENE_PRUNE_EMISSIVE)
        try:
            found = scene.emissive()
            st.emissive[: found.size] = found
            st.emissive[found.size:] = -1
            return st.emissive
        finally:
            scene.close()
    env = Env(ctx, st.sky)
    try:
        return list(env.cdf())
    finally:
        env.close()


# -------------------------------------------------------------------- work
def _paths_work(paths, edge, bounces):
    """Operations of `paths` samples in a volume of that edge: a segment crosses about a tenth of the volume's cells
    along its way at seven operations a cell, and a shaded vertex takes about six hundred."""
    segments = 1.0 + 1.7 * min(bounces, 2)
    return paths * (segments * 0.1 * edge * 7.0 + min(bounces, 2) * 600.0 + 150.0)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        voxels = case["rx"] * case["ry"] * case["rz"]
        edge = voxels ** (1.0 / 3.0)
        pixels = case["w"] * case["h"]
        # occupancy is one bit a voxel; the palette bytes of what the rays meet are few
        return {"bytes": voxels / 8 + 8 * case["env_w"] * case["env_h"] + 16 * pixels,
                "flops": _paths_work(pixels * case["spp"], edge, case["bounces"])}
    if kind in ("batch", "serve"):
        edge = math.sqrt(case["edge_min"] * case["edge_max"])
        pixels = 260.0 ** 2 * case["jobs"]
        spp = case["spp"] if kind == "batch" else 0.45 * case["spp"]
        return {"bytes": case["jobs"] * edge ** 3 / 8 + 16 * pixels,
                "flops": _paths_work(pixels * spp, edge, case["bounces"])}
    if kind == "mesh":
        voxels = case["rx"] * case["ry"] * case["rz"]
        tris = 4 * case["rows"] ** 2
        pixels = case["w"] * case["h"]
        return {"bytes": voxels + 12 * tris + 6 * tris + 16 * pixels,
                "flops": 300.0 * tris + 7.0 * pixels * voxels ** (1.0 / 3.0)}
    if kind == "load":
        voxels = case["rx"] * case["ry"] * case["rz"]
        return {"bytes": 2 * voxels + voxels / 8, "flops": 1.0 * voxels}
    texels = case["env_w"] * case["env_h"]
    return {"bytes": 12 * texels + 8 * texels + 4 * texels, "flops": 30.0 * texels}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The environment's CDFs and integral in 64 bits: FP16 texels, Rec.709 luminance, a three-tap Gaussian blur of
    sigma 0.75 px clamped at the edges, sin(theta) weights, prefix sums by rows and over the rows."""
    if case["kind"] != "env":
        return None
    rgb = np.clip(_sky(case["env_w"], case["env_h"], seed), -65504.0, 65504.0).astype(np.float16).astype(np.float64)
    lum = rgb @ np.array([0.2126, 0.7152, 0.0722])
    e = math.exp(-1.0 / (2.0 * 0.75 ** 2))
    side, mid = e / (1.0 + 2.0 * e), 1.0 / (1.0 + 2.0 * e)
    for axis in (1, 0):
        p = np.pad(lum, [(0, 0), (1, 1)] if axis == 1 else [(1, 1), (0, 0)], mode="edge")
        n = lum.shape[axis]
        lum = side * np.take(p, range(n), axis) + mid * lum + side * np.take(p, range(2, n + 2), axis)
    h, w = lum.shape
    f = np.maximum(0.0, lum) * np.sin(math.pi * (np.arange(h) + 0.5) / h)[:, None]
    rows = np.concatenate([np.zeros((h, 1)), np.cumsum(f, 1)], 1)
    total = rows[:, -1:]
    cdf_u = np.where(total > 0.0, rows / np.where(total > 0.0, total, 1.0), np.arange(w + 1)[None, :] / w)
    marginal = np.concatenate([[0.0], np.cumsum(total[:, 0] / w)])
    return [cdf_u, marginal / marginal[-1], float(marginal[-1] / h * 2.0 * math.pi ** 2)]
