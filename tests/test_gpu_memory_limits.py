"""Renders and builds where device memory is short: on the device, and under a
context's budget."""
import numpy as np
import pytest

from helpers import close_all, gpu_setup, small_config2
from voxeltoy_gb300 import Context, Job, Scene
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu

PALETTE = [S.lambert(0.7)]


def open_volume(edge):
    vox = np.zeros((edge,) * 3, np.uint8)
    vox[0, 0, 0] = vox[-1, -1, -1] = vox[edge // 2, edge // 2, edge // 2] = 1
    return vox


@pytest.mark.parametrize("integrator", [0, 1])
def test_a_render_goes_on_where_free_cubes_find_no_memory(integrator):
    """The renders of an open scene on a device without room for its free cubes
    succeed without them, and count their samples."""
    torch = pytest.importorskip("torch")
    vox = open_volume(512)
    cam, s = S.orbit_camera(distance=500.0), S.physical_settings(3, seed=4)
    with Context() as ctx:
        a, b = (Scene.dense(ctx, vox, PALETTE) for _ in range(2))
        jobs = [Job(ctx, sc, None, cam, s, 64, 48) for sc in (a, b)]
        held = []
        try:
            before = b.info().device_bytes
            for j in jobs:
                j.set_integrator(integrator)
            for _ in range(2):                     # its kernels are loaded, its buffers there
                jobs[0].render(1)
            want = jobs[0].readback()
            jobs[1].readback()
            assert a.info().device_bytes > before
            ctx.trim()
            size = torch.cuda.mem_get_info()[0]
            while size >= 1 << 21:                 # the rest of the device, down to 2 MB
                try:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.cuda.OutOfMemoryError:
                    size //= 2
            for _ in range(2):
                jobs[1].render(1)
            assert jobs[1].samples() == 2 and b.info().device_bytes == before
            assert np.array_equal(jobs[1].readback().view(np.uint32), want.view(np.uint32))
        finally:
            held.clear()
            torch.cuda.empty_cache()
            close_all(*jobs, a, b)


def test_block_wavefront_state_gives_way_under_a_budget():
    """What a launch as block wavefronts keeps for the next one counts against
    the budget, and is given up for a scene, a job or a readback that needs it;
    the next launch then is the wavefront, with the few path slots that fit."""
    cfg = small_config2(edge=24, w=400, h=401, seed=11)
    vox = open_volume(200)
    used = 0
    for budget in (0, 1):
        with Context(0, hbm_budget_bytes=budget and used) as ctx:
            ctx.set_tuning(path_slots=1024)
            scene, env, job = gpu_setup(ctx, cfg)
            more = []
            try:
                job.render(1)
                used = ctx.memory() + (1 << 20)    # a MB beside what the render keeps
                if budget:
                    image = job.readback()         # a buffer of 2.6 MB
                    more.append(Scene.dense(ctx, vox, PALETTE))                            # 8 MB
                    more.append(Job(ctx, more[0], None, cfg.camera, cfg.settings, 400, 400))   # 5 MB
                    job.render(1)
                    assert job.samples() == 2
                else:
                    want = job.readback()
            finally:
                close_all(*more[::-1], job, scene, env)
    assert np.array_equal(image.view(np.uint32), want.view(np.uint32))


def test_device_bytes_count_the_free_cubes():
    """The first render of an open scene adds eight bytes a padded brick."""
    with Context() as ctx:
        scene = Scene.dense(ctx, open_volume(96), PALETTE)
        job = Job(ctx, scene, None, S.orbit_camera(), S.physical_settings(2), 32, 32)
        try:
            before, held = scene.info().device_bytes, ctx.memory()
            for _ in range(2):
                job.render(1)
                assert scene.info().device_bytes == before + 8 * 26 ** 3
            assert ctx.memory() - held >= 8 * 26 ** 3
            scene.set_brick_shape((1, 2, 3))
            job.render(1)
            scene.set_brick_shape((2, 2, 2))
            assert scene.info().device_bytes == before
        finally:
            close_all(job, scene)


@pytest.mark.parametrize("edge,w,h,passes,built", [(96, 64, 48, 1, 2), (96, 1024, 1024, 2, 1), (640, 64, 48, 1, 1)])
def test_a_first_edit_mode_image_leaves_the_free_cubes_to_the_second(edge, w, h, passes, built):
    """A scene's first edit-mode image builds free cubes where the volume or the
    call is large, any other image does, and all are the same without them."""
    with Context() as ctx:
        scenes = [Scene.dense(ctx, open_volume(edge), PALETTE) for _ in range(3)]
        jobs = [Job(ctx, sc, None, S.orbit_camera(distance=700.0), S.physical_settings(2), w, h) for sc in scenes]
        try:
            scenes[1].set_brick_shape((1, 2, 3))
            bytes_ = [sc.info().device_bytes for sc in scenes]
            for n in (1, 2, 3):
                for j in jobs[:2]:
                    j.set_integrator(1)
                    j.render(passes)
                assert (scenes[0].info().device_bytes > bytes_[0]) == (n >= built)
                a, b = (j.readback().view(np.uint32) for j in jobs[:2])
                assert np.array_equal(a, b)
            jobs[2].render(1)                              # the path tracer's first image
            assert scenes[2].info().device_bytes > bytes_[2]
        finally:
            close_all(*jobs, *scenes)
