"""The forms a launch takes by its number of samples (a thread per sample, block
wavefronts, the wavefront): every form gives the wavefront's image bit for bit,
on both sides of each size where the form changes, for one job, a parameter
table of jobs and a global one, ragged volumes, other brick shapes, the noise
table, and rays that miss the volume.  The wavefront itself is compared with
the oracle in test_gpu_parity.py."""
import numpy as np
import pytest

from helpers import close_all, gpu_setup, reference_config, small_config1, small_config2
from voxeltoy_gb300 import Context, Job

pytestmark = pytest.mark.gpu

PATHS = 1 << 17             # kPathsItems
BLOCK = (16 << 20) // 10    # kBlockWork over the rounds of eight bounces: 1677721


@pytest.fixture(scope="module")
def fctx():
    c = Context()
    yield c
    c.close()


def compare(ctx, cfgs, passes, shape=None):
    """Every job rendered in one call by size and by the wavefront."""
    made = [gpu_setup(ctx, c) for c in cfgs]
    refs = [Job(ctx, s, e, c.camera, c.settings, c.width, c.height) for (s, e, _j), c in zip(made, cfgs)]
    jobs = [m[2] for m in made]
    try:
        if shape:
            for m in made:
                m[0].set_brick_shape(shape)
        for _ in range(2):                       # the second call continues the accumulation
            ctx.render_batch(jobs, passes)
            ctx.render_batch(refs, passes, kernel=2)
        for j, r in zip(jobs, refs):
            assert j.samples() == r.samples()
            a, b = j.readback(), r.readback()
            same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))   # NaN payloads aside
            assert same.all()
    finally:
        close_all(*refs)
        for s, e, j in made:
            close_all(j, s, e)


def config2(w, h, edge=24, seed=11):
    cfg = small_config2(edge=edge, w=w, h=h, seed=seed)
    cfg.settings.max_samples = 1 << 20
    return cfg


@pytest.mark.parametrize("w,h,passes", [
    (1, 1, 1), (1, 1, 33), (31, 1, 2), (33, 7, 5),             # a thread per sample
    (512, 256, 1), (512, 257, 1), (256, 128, 4),               # PATHS, past it
    (1024, 819, 2), (1024, 820, 2), (701, 499, 3),             # BLOCK, past it, between
])
def test_forms_agree_at_their_limits(fctx, w, h, passes):
    compare(fctx, [config2(w, h)], passes)


@pytest.mark.parametrize("n_jobs", [2, 8, 9, 17])
@pytest.mark.parametrize("scale", [1, 6])
def test_forms_agree_for_several_jobs(fctx, n_jobs, scale):
    cfgs = []
    for k in range(n_jobs):
        make = config2 if k % 2 else (lambda w, h, edge, seed: small_config1(edge=edge, w=w, h=h, seed=seed))
        cfg = make((17 + 9 * k) * scale, (23 + 3 * k) * scale, edge=20 + 5 * (k % 4), seed=20 + k)
        cfg.settings.max_samples = 1 << 20
        cfgs.append(cfg)
    compare(fctx, cfgs, 2)


@pytest.mark.parametrize("shape", [(1, 2, 3), (4, 1, 1), (2, 2, 2)])
@pytest.mark.parametrize("w,h", [(40, 28), (400, 401)])
def test_forms_agree_for_every_brick_shape_and_the_noise_table(fctx, shape, w, h):
    a = config2(w, h, edge=37)
    b = reference_config(w=w, h=h)
    b.settings.max_samples = 1 << 20
    a.voxels = np.ascontiguousarray(a.voxels[:29, :, :33])     # a ragged volume
    compare(fctx, [a, b], 2, shape=shape)


@pytest.mark.parametrize("w,h", [(64, 48), (600, 500)])
def test_forms_agree_where_most_rays_miss(fctx, w, h):
    cfg = config2(w, h)
    for i in range(3):
        cfg.camera.eye[i] = cfg.camera.eye[i] * 6.0
    compare(fctx, [cfg], 3)


@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (8, 4), (33, 65), (160, 121), (301, 203), (512, 300)])
def test_edit_mode_images_are_their_samples(fctx, w, h):
    """Edit-mode images, rendered in tiles of 8 x 1, 2 or 4 pixels by size,
    against the samples that the pixel-per-thread diagnostic gives (compared
    with the oracle elsewhere)."""
    cfg = config2(w, h)
    cfg.settings.wireframe_opacity = 0.6
    scene, env, job = gpu_setup(fctx, cfg)
    try:
        job.set_integrator(1)
        want = job.samples_diag(0)[0]
        job.render(1)
        assert np.array_equal(job.readback().view(np.uint32), want.view(np.uint32))
        job.render(2)
        assert job.samples() == 3
    finally:
        close_all(job, scene, env)


def test_small_budgets_take_the_wavefront():
    """A budget that holds the wavefront with few path slots, but not the block
    form's state, still renders, and the same image; so does a wavefront launch
    that needs the memory an earlier block launch kept."""
    cfg = config2(400, 401)                    # block form: 160400 samples
    big = config2(1200, 1000)                  # the wavefront by size
    images = []
    for budget in (0, 24 << 20):       # the block form wants 30 MB in all, the wavefront 9
        with Context(0, hbm_budget_bytes=budget) as ctx:
            ctx.set_tuning(path_slots=1024)
            made = gpu_setup(ctx, cfg)
            job = made[2]
            try:
                job.render(1)
                images.append(job.readback())
            finally:
                close_all(made[2], made[0], made[1])
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
    images = []
    for budget in (0, 204 << 20):      # 197 MB, and 22 that the block form keeps
        with Context(0, hbm_budget_bytes=budget) as ctx:
            a, b = gpu_setup(ctx, cfg), gpu_setup(ctx, big)
            try:
                a[2].render(1)
                ctx.set_tuning(path_slots=300000)
                b[2].render(2)
                close_all(a[2], a[0], a[1])    # their memory is what the readback's buffer takes
                a = (None, None, None)
                images.append(b[2].readback())
            finally:
                close_all(a[2], a[0], a[1], b[2], b[0], b[1])
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
