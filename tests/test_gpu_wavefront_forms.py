"""The wavefront's own forms, asked for by name (kernel 2) whatever a launch's
size would choose, with the number of kernels launched as the evidence of the
form: groups of rounds launched directly or replayed, lanes, DDA kernel forms;
and the way back to a context's defaults."""
import numpy as np
import pytest

from helpers import close_all, gpu_setup, small_config2
from voxeltoy_gb300 import Context, Job, Scene
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture
def wctx():
    c = Context()
    yield c
    c.close()


def config(w, h, bounces=8, edge=24, seed=15):
    cfg = small_config2(edge=edge, w=w, h=h, seed=seed)
    cfg.settings.max_samples = 1 << 20
    cfg.settings.max_bounces = bounces
    return cfg


def frame(ctx, job, passes, **kw):
    """The image's words and the kernels launched for it."""
    job.reset()
    n = ctx.launch_count()
    ctx.render_batch([job], passes, kernel=2, **kw)
    n = ctx.launch_count() - n
    return job.readback().view(np.uint32).copy(), n


def group(lanes, rounds):
    return lanes * rounds * 4      # shade, hit, regen and trace, a lane and round


@pytest.mark.parametrize("lanes", [1, 2, 3, 4])
@pytest.mark.parametrize("w,h,passes", [(641, 479, 1), (641, 479, 3), (150, 131, 1), (256, 256, 2)])
def test_samples_with_a_slot_each_take_one_group(wctx, lanes, w, h, passes):
    """Launches whose samples all fit the path slots run max_bounces + 2 rounds
    (made even) once, whatever the sample count leaves when divided by the lanes."""
    scene, env, job = gpu_setup(wctx, config(w, h))
    try:
        wctx.set_lanes(lanes)
        got, n = frame(wctx, job, passes)
        assert n == group(lanes, 10) + 1
        job.reset()
        wctx.render_batch([job], passes, kernel=1)
        assert np.array_equal(got, job.readback().view(np.uint32))
    finally:
        close_all(job, scene, env)


@pytest.mark.parametrize("lanes", [1, 2, 3, 4])
def test_replayed_groups_equal_direct_ones(wctx, lanes):
    """Rounds replayed from a graph against the same rounds launched one by one,
    with fewer slots than samples, so that both take several groups."""
    scene, env, job = gpu_setup(wctx, config(96, 80))
    try:
        wctx.set_lanes(lanes)
        images, counts = [], []
        for graphs in (True, False, True):
            wctx.set_graphs(graphs)
            a, n = frame(wctx, job, 5, path_slots=4096)
            images.append(a)
            counts.append(n)
        assert counts[0] == counts[1] == counts[2] > 2 * group(lanes, 8)
        assert np.array_equal(images[0], images[1]) and np.array_equal(images[0], images[2])
    finally:
        close_all(job, scene, env)


def test_lanes_agree(wctx):
    scene, env, job = gpu_setup(wctx, config(96, 80))
    try:
        images = []
        for lanes in (1, 2, 3, 4):
            wctx.set_lanes(lanes)
            for slots, rounds in ((0, 10), (4096, 8)):
                a, n = frame(wctx, job, 3, path_slots=slots)
                assert (n - 1) % group(lanes, rounds) == 0
                images.append(a)
        for a in images[1:]:
            assert np.array_equal(a, images[0])
    finally:
        close_all(job, scene, env)


@pytest.mark.parametrize("slots", [0, 4096])
@pytest.mark.parametrize("open_scene", [False, True])
def test_trace_forms_agree(wctx, slots, open_scene):
    cfg = config(96, 80)
    if open_scene:
        cfg.voxels = np.zeros((96, 90, 84), np.uint8)
        cfg.voxels[10:14, ::7, ::5] = 1
    scene, env, job = gpu_setup(wctx, cfg)
    try:
        images = []
        for form in (0, 1):
            wctx.set_trace_form(form)
            for steps in (4, 8, 16):
                wctx.set_tuning(trace_steps=steps)
                images.append(frame(wctx, job, 3, path_slots=slots)[0])
        for a in images[1:]:
            assert np.array_equal(a, images[0])
    finally:
        close_all(job, scene, env)

def test_back_to_the_defaults(wctx):
    """The kernel form and the DDA steps return to the choice by size and by
    volume; other values are refused."""
    scene, env, job = gpu_setup(wctx, config(32, 32))
    try:
        images = []
        for kernel, kernels in ((0, 1), (1, 1), (2, group(1, 10) + 1), (0, 1)):
            wctx.set_kernel(kernel)
            wctx.set_tuning(trace_steps=32 if kernel else L.VT_DIAG_TRACE_STEPS_AUTO)
            job.reset()
            n = wctx.launch_count()
            job.render(1)
            assert wctx.launch_count() - n == kernels
            images.append(job.readback().view(np.uint32).copy())
        for a in images[1:]:
            assert np.array_equal(a, images[0])
        for bad in (-1, 3):
            with pytest.raises(L.VtError):
                wctx.set_kernel(bad)
    finally:
        close_all(job, scene, env)

@pytest.mark.parametrize("w,h,bounces,inside,block", [
    (768, 512, 3, True, True), (769, 512, 3, True, False), (769, 512, 3, False, True), (480, 270, 3, True, True),
    (768, 512, 2, True, True), (769, 512, 2, True, False), (1024, 768, 1, True, True), (1025, 768, 1, True, False),
    (1536, 1024, 0, True, True), (1537, 1024, 0, True, False), (769, 512, 64, False, False), (513, 300, 64, True, True)])
def test_cameras_inside_the_volume_leave_the_block_form_earlier(wctx, w, h, bounces, inside, block):
    """A launch by size takes one kernel and the accumulation (a single pass of
    few samples one kernel), or the wavefront's; the images are the same."""
    cfg = config(w, h, bounces=bounces)
    if inside:
        cfg.voxels = np.ones((24, 24, 24), np.uint8)
        cfg.voxels[3:-3, 3:-3, 3:-3] = 0
        cfg.voxels[20, 21, 10:14] = 2
        cfg.camera = S.orbit_camera(distance=150.0)
    scene, env, job = gpu_setup(wctx, cfg)
    other = Job(wctx, scene, env, cfg.camera, cfg.settings, 40, 30)
    try:
        want, rounds = frame(wctx, job, 1)
        job.reset()
        n = wctx.launch_count()
        job.render(1)
        n = wctx.launch_count() - n
        assert n == ((1 if w * h <= 1 << 17 else 2) if block else rounds)
        assert np.array_equal(job.readback().view(np.uint32), want)
        job.reset()
        n = wctx.launch_count()
        wctx.render_batch([job, other], 1, kernel=2)
        n_all = wctx.launch_count() - n
        job.reset()
        other.reset()
        n = wctx.launch_count()
        wctx.render_batch([job, other], 1)            # both cameras count
        n = wctx.launch_count() - n
        line = max(3 << 17, (3 << 19) >> bounces) if inside else 1 << 30
        small = (w * h + 1200) * (bounces + 2) <= 16 << 20
        assert n == (2 if small and w * h + 1200 <= min(line, (bounces + 2) << 18) else n_all)
        assert np.array_equal(job.readback().view(np.uint32), want)
    finally:
        close_all(other, job, scene, env)

def test_tuning_times_the_wavefront_and_leaves_the_form(wctx):
    """A small job's sweep launches wavefronts; afterwards its renders take the
    form by size again."""
    from voxeltoy_gb300 import autotune
    scene, env, job = gpu_setup(wctx, config(32, 32))
    try:
        n = wctx.launch_count()
        best = autotune.tune(wctx, [job], passes=1, repeats=1, use_cache=False,
                             grid={"path_slots": [1 << 20], "trace_blocks_per_sm": [0], "trace_steps": [8, 16],
                                   "lanes": [1], "brick_shape": [(2, 2, 2)], "queue_chunk": [64], "refill_min": [0]})
        assert wctx.launch_count() - n >= (group(1, 10) + 1) * len(best["sweep"]) * best["repeats"]
        n = wctx.launch_count()
        job.render(1)
        assert wctx.launch_count() - n == 1
    finally:
        close_all(job, scene, env)


@pytest.mark.parametrize("w,h,jobs,block", [(512, 512, 2, True), (512, 513, 2, False), (1024, 513, 1, True), (256, 256, 8, True),
                                            (256, 257, 8, False)])
def test_several_jobs_leave_the_block_form_earlier(wctx, w, h, jobs, block):
    """Launches of several jobs take the block form up to 2^18 samples a round
    (two rounds here); the images are the wavefront's."""
    made = [gpu_setup(wctx, config(w, h, bounces=0, seed=30 + k)) for k in range(jobs)]
    js = [m[2] for m in made]
    try:
        wctx.render_batch(js, 1, kernel=2)
        want = [j.readback().view(np.uint32) for j in js]
        for j in js:
            j.reset()
        n = wctx.launch_count()
        wctx.render_batch(js, 1)
        n = wctx.launch_count() - n
        assert n == 2 if block else n > 8
        for j, a in zip(js, want):
            assert np.array_equal(j.readback().view(np.uint32), a)
    finally:
        for sc, env, j in made:
            close_all(j, sc, env)
