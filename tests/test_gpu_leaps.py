"""Free cubes and the DDA's leaps through them: images with 4x4x4 bricks
(leaps) equal images with another brick shape (no leaps) bit for bit, in nearly
empty, ragged and edited volumes, for every launch form and integrator, with
rays along the axes and diagonals (ties) among them."""
import numpy as np
import pytest

from helpers import close_all
from voxeltoy_gb300 import Context, Job, Scene
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fctx():
    c = Context()
    yield c
    c.close()


def volume(kind, res, seed=1):
    rx, ry, rz = res
    z, y, x = np.mgrid[0:rz, 0:ry, 0:rx].astype(np.float32)
    g = np.zeros((rz, ry, rx), np.uint8)
    rng = np.random.default_rng(seed)
    if kind == "shell":
        r = np.sqrt(((x - rx / 2) / rx) ** 2 + ((y - ry / 2) / ry) ** 2 + ((z - rz / 2) / rz) ** 2)
        g[np.abs(r - 0.4) < 0.006] = 1
    elif kind == "dust":           # single voxels far apart
        n = max(3, g.size // 20000)
        g[rng.integers(0, rz, n), rng.integers(0, ry, n), rng.integers(0, rx, n)] = 1
    elif kind == "slab":
        g[:, 0, :] = 1
    g[rng.integers(0, rz), rng.integers(0, ry), rng.integers(0, rx)] = 2
    return g


def cameras():
    out = [S.orbit_camera(theta_deg=110.0, phi_deg=37.0), S.orbit_camera(distance=700.0, theta_deg=95.0, phi_deg=200.0)]
    for theta, phi in ((90.0, 0.0), (125.2643897, 45.0), (120.0, 30.0)):   # along z, the diagonal, oblique
        cam = S.orbit_camera(theta_deg=theta, phi_deg=phi, lens=L.VT_LENS_ORTHOGRAPHIC)
        out.append(cam)
    return out


PALETTE = [S.lambert(0.7), S.lambert(0.3, emission=(4.0, 3.0, 2.0)), S.metal(0.8, 0.2)]


def images(ctx, scene, w, h, passes, kernels=(0, 1, 2), integrators=(0, 1)):
    out = []
    for cam in cameras():
        for integ in integrators:
            for kernel in kernels:
                s = S.physical_settings(5, seed=3, top=(1.0, 0.9, 0.8), bottom=(0.3, 0.4, 0.5))
                job = Job(ctx, scene, None, cam, s, w, h)
                try:
                    job.set_integrator(integ)
                    ctx.render_batch([job], passes, kernel=kernel)
                    out.append(job.readback().copy())
                finally:
                    job.close()
    return out


def same(a, b):
    for p, q in zip(a, b):
        assert np.array_equal(p.view(np.uint32), q.view(np.uint32))


@pytest.mark.parametrize("res", [(64, 64, 64), (131, 70, 93), (40, 300, 33), (257, 129, 260)])
@pytest.mark.parametrize("kind", ["shell", "dust", "slab"])
def test_leaps_change_no_pixel(fctx, res, kind):
    vox = volume(kind, res)
    a = Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE)
    b = Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE)
    try:
        b.set_brick_shape((1, 2, 3))
        before = a.info().device_bytes
        same(images(fctx, a, 61, 47, 2), images(fctx, b, 61, 47, 2))
        if min(res) > 64 and kind != "shell":      # open enough to hold free cubes
            assert a.info().device_bytes > before
    finally:
        close_all(a, b)


def test_leaps_where_the_cubes_are_built_in_long_runs(fctx):
    """A volume of more than 2^18 bitmap words, whose cubes' slices are taken
    eight at a time, with a last run that is not full."""
    rng = np.random.default_rng(5)
    vox = np.zeros((2059, 2061, 24), np.uint8)
    vox[rng.integers(0, 2059, 3000), rng.integers(0, 2061, 3000), rng.integers(0, 24, 3000)] = 1
    a, b = (Scene.dense(fctx, vox, PALETTE) for _ in range(2))
    try:
        b.set_brick_shape((1, 2, 3))
        before = a.info().device_bytes
        same(images(fctx, a, 61, 47, 2), images(fctx, b, 61, 47, 2))
        assert a.info().device_bytes > before
    finally:
        close_all(a, b)


@pytest.mark.parametrize("size", [(400, 401), (1024, 800)])
def test_leaps_in_larger_launches(fctx, size):
    vox = volume("shell", (200, 180, 220))
    a, b = (Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE) for _ in range(2))
    try:
        b.set_brick_shape((3, 2, 1))
        same(images(fctx, a, *size, 4, kernels=(0,), integrators=(0,)), images(fctx, b, *size, 4, kernels=(0,), integrators=(0,)))
    finally:
        close_all(a, b)


def test_edits_keep_free_cubes_bounds(fctx):
    """Voxels set in the middle of free cubes after these were built, then
    emptied again: every image equals that of a scene built from the result."""
    res = (150, 141, 133)
    vox = volume("slab", res)
    sc = Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE)
    rng = np.random.default_rng(8)
    try:
        images(fctx, sc, 8, 8, 1)                       # builds the free cubes
        spots = [(int(rng.integers(0, res[0])), int(rng.integers(0, res[1])), int(rng.integers(0, res[2])))
                 for _ in range(12)] + [(0, 140, 0), (149, 140, 132), (75, 70, 66)]
        for entry in (1, 0):
            for x, y, z in spots if entry else spots[::2]:
                sc.set_voxel(x, y, z, entry)
                vox[z, y, x] = entry
            ref = Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE)
            ref.set_brick_shape((1, 2, 3))
            try:
                same(images(fctx, sc, 53, 41, 2), images(fctx, ref, 53, 41, 2))
            finally:
                ref.close()
    finally:
        sc.close()


def test_brick_shape_and_back(fctx):
    vox = volume("dust", (90, 80, 70))
    sc = Scene.dense(fctx, vox, PALETTE)
    try:
        a = images(fctx, sc, 40, 30, 1)
        sc.set_brick_shape((4, 1, 1))
        same(a, images(fctx, sc, 40, 30, 1))
        sc.set_brick_shape((2, 2, 2))
        same(a, images(fctx, sc, 40, 30, 1))
    finally:
        sc.close()


def test_no_free_cubes_under_a_budget():
    vox = volume("dust", (90, 80, 70))
    with Context(0, hbm_budget_bytes=64 << 20) as ctx:
        sc = Scene.dense(ctx, vox, PALETTE)
        job = Job(ctx, sc, None, cameras()[0], S.physical_settings(3), 32, 32)
        try:
            before = sc.info().device_bytes
            job.render(1)
            assert sc.info().device_bytes == before
        finally:
            close_all(job, sc)
