"""Scenes used by more than one stream: a server that renders a caller's scene
while the caller's context is at work or edits it, jobs on one context that
render another context's scene, and tables replaced behind a render."""
import time

import numpy as np
import pytest

from helpers import close_all
from voxeltoy_gb300 import Context, Job, Scene, Server
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu

PALETTE = [S.lambert(0.95), S.lambert(0.0), S.lambert(0.5, emission=(6.0, 5.0, 4.0))]


@pytest.fixture
def sctx():
    c = Context()
    yield c
    c.close()


def room_job(ctx, room, w=64, h=64, rng_mode=L.VT_RNG_PHILOX):
    """A job whose passes take milliseconds: up to 1024 bounces between the walls."""
    s = S.physical_settings(1024, seed=5)
    s.rng_mode = rng_mode
    return Job(ctx, room, None, S.orbit_camera(distance=120.0), s, w, h)


def make_room(ctx, edge=8):
    vox = np.ones((edge,) * 3, np.uint8)
    vox[1:-1, 1:-1, 1:-1] = 0
    lights = [(edge - 1, y, x) for y in (2, 4) for x in (2, 5)]
    for at in lights:
        vox[at] = 3
    emissive = np.array([x + edge * (y + edge * z) for z, y, x in lights], np.int32)
    return Scene.dense(ctx, vox, PALETTE, emissive=emissive)


def queue_work(ctx, job, seconds=1.0):
    """About that much GPU time on the context's stream, queued without waiting."""
    ctx.render_batch([job], 1, kernel=1)
    job.synchronize()
    t0 = time.perf_counter()
    ctx.render_batch([job], 4, kernel=1)
    job.synchronize()
    passes = int(min(800, max(4, 4 * seconds / (time.perf_counter() - t0))))
    ctx.render_batch([job], passes, kernel=1)


def open_volume(edge=96):
    """Nearly all of it free cubes, a little matter in the corners."""
    vox = np.zeros((edge,) * 3, np.uint8)
    vox[0, 0, 0] = vox[-1, -1, -1] = vox[0, -1, 0] = 1
    return vox


def image(ctx, scene, edge=64):
    job = Job(ctx, scene, None, S.orbit_camera(distance=300.0), S.physical_settings(3, seed=2), edge, edge)
    try:
        job.render(2)
        return job.readback()
    finally:
        job.close()


def test_edit_beside_a_servers_first_render(sctx):
    """A voxel set by the owner while a server renders the scene for the first
    time is there in every later image."""
    room = make_room(sctx)
    busy = room_job(sctx, room)
    vox = open_volume()
    warm, scene = Scene.dense(sctx, vox, PALETTE), Scene.dense(sctx, vox, PALETTE)
    srv = Server(sctx)
    cam, settings = S.orbit_camera(distance=300.0), S.physical_settings(3)
    try:
        assert srv.wait(srv.submit(warm, None, cam, settings, 32, 32, 1), 60.0) == L.VT_OK
        queue_work(sctx, busy)
        ticket = srv.submit(scene, None, cam, settings, 32, 32, 1)
        time.sleep(0.3)
        scene.set_voxel(48, 48, 48, 1)
        vox[48, 48, 48] = 1
        assert srv.wait(ticket, 60.0) == L.VT_OK
        ref = Scene.dense(sctx, vox, PALETTE)
        ref.set_brick_shape((1, 2, 3))
        try:
            assert np.array_equal(image(sctx, scene).view(np.uint32), image(sctx, ref).view(np.uint32))
        finally:
            ref.close()
    finally:
        srv.close()
        close_all(busy, room, warm, scene)


def test_servers_first_render_leaves_the_owners_stream_alone(sctx):
    """A server's first render of a scene finishes while its owner's stream is
    still at work."""
    room = make_room(sctx)
    busy = room_job(sctx, room)
    warm, scene = (Scene.dense(sctx, open_volume(), PALETTE) for _ in range(2))
    srv = Server(sctx)
    cam, settings = S.orbit_camera(distance=300.0), S.physical_settings(3)
    try:
        assert srv.wait(srv.submit(warm, None, cam, settings, 32, 32, 1), 60.0) == L.VT_OK
        before = scene.info().device_bytes
        queue_work(sctx, busy, 2.0)
        ticket = srv.submit(scene, None, cam, settings, 32, 32, 1)
        assert srv.wait(ticket, 60.0) == L.VT_OK
        t0 = time.perf_counter()
        busy.synchronize()
        assert time.perf_counter() - t0 > 0.3
        assert scene.info().device_bytes > before         # with free cubes
    finally:
        srv.close()
        close_all(busy, room, warm, scene)


def test_owner_renders_beside_servers_first_renders(sctx):
    """Launches that the owner replays as a graph go on, and give the same
    image, while a server renders the owner's scenes for the first time."""
    room = make_room(sctx, 24)
    s = S.physical_settings(8, seed=5)
    job = Job(sctx, room, None, S.orbit_camera(distance=120.0), s, 64, 64)
    scenes = [Scene.dense(sctx, open_volume(64), PALETTE) for _ in range(40)]
    srv = Server(sctx)
    cam, settings = S.orbit_camera(distance=300.0), S.physical_settings(3)

    def frame():
        job.reset()
        sctx.render_batch([job], 8, kernel=2, path_slots=1024)
        return job.readback().view(np.uint32)
    try:
        want = frame()
        for scene in scenes:
            ticket = srv.submit(scene, None, cam, settings, 16, 16, 1)
            while True:
                assert np.array_equal(frame(), want)
                if srv.poll(ticket)[0] not in (0, 1):     # queued, running
                    break
            assert srv.wait(ticket, 60.0) == L.VT_OK
    finally:
        srv.close()
        close_all(job, room, *scenes)


def test_edit_after_a_render_on_another_context(sctx):
    """A job on one context renders another context's scene; an edit of the
    scene after the call is not in its image."""
    room = make_room(sctx)
    with Context() as other:
        job = room_job(other, room)
        try:
            job.render(1)
            job.synchronize()
            want = job.readback()
            job.reset()
            job.synchronize()
            job.render(1)
            for y in range(1, 7):
                for z in range(1, 7):
                    room.set_voxel(0, y, z, 2)            # a white wall turns black
            assert np.array_equal(job.readback().view(np.uint32), want.view(np.uint32))
            job.reset()
            job.render(1)
            assert not np.array_equal(job.readback().view(np.uint32), want.view(np.uint32))
        finally:
            job.close()
    room.close()


def test_noise_table_replaced_after_a_render(sctx):
    """A render uses the noise table of its call."""
    room = make_room(sctx)
    job = room_job(sctx, room, rng_mode=L.VT_RNG_NOISE_TABLE)
    table = sctx.noise_table()
    other = np.ascontiguousarray(table[::-1, ::-1])
    put = lambda t: L.call("vt_diag_set_noise_table", sctx.h, L.ptr(t), t.nbytes)
    try:
        job.render(1)
        want = job.readback()
        for _ in range(4):
            job.reset()
            job.synchronize()
            job.render(1)
            put(other)
            assert np.array_equal(job.readback().view(np.uint32), want.view(np.uint32))
            put(table)
        put(other)
        job.reset()
        job.render(1)
        assert not np.array_equal(job.readback().view(np.uint32), want.view(np.uint32))
    finally:
        close_all(job, room)
