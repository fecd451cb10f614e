"""The autotuner times the kernels that its knobs set, whatever form a launch
of the timed size would take by itself, and puts the context's choice back."""
import pytest

from test_autotune import FakeCtx, FakeJob, fake_time  # noqa: F401
from voxeltoy_gb300 import autotune


class FormCtx(FakeCtx):
    """A context whose default form knows none of the knobs."""

    def __init__(self, kernel=0):
        super().__init__()
        self.kernel = kernel
        self.kernels = []

    def set_kernel(self, kernel):
        self.kernel = kernel
        self.kernels.append(kernel)


class FormJob(FakeJob):
    def render(self, passes):
        if self.ctx.kernel == 2:
            super().render(passes)
        else:
            self.clock[0] += 0.1 * passes * self.unit


@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_the_wavefront_is_timed_and_the_form_put_back(fake_time, kernel):  # noqa: F811
    ctx = FormCtx(kernel)
    job = FormJob(ctx, fake_time, w=4096, h=4096)
    best = autotune.tune(ctx, [job], repeats=1, use_cache=False)
    assert (best["path_slots"], best["trace_blocks_per_sm"], best["trace_steps"], best["lanes"]) == (1 << 23, 3, 16, 2)
    assert len({r["seconds"] for r in best["sweep"]}) > 10        # not one time for every setting
    assert ctx.kernels[0] == 2 and ctx.kernel == kernel


def test_the_form_is_put_back_after_an_error(fake_time):  # noqa: F811
    class Failing(FormJob):
        def render(self, passes):
            if self.renders == 5:
                raise RuntimeError("lost")
            super().render(passes)

    ctx = FormCtx()
    with pytest.raises(RuntimeError):
        autotune.tune(ctx, [Failing(ctx, fake_time, w=4096, h=4096)], repeats=1, use_cache=False)
    assert ctx.kernel == 0


def test_the_key_holds_the_samples_and_the_form(fake_time):  # noqa: F811
    a = FakeJob(FakeCtx(), [0.0], w=512, h=512)
    assert autotune.workload_key([a], 1) != autotune.workload_key([a], 64)
    ctx = FormCtx()
    job = FormJob(ctx, fake_time, w=64, h=64)
    keys = [autotune.tune(ctx, [job], passes=p, repeats=1, use_cache=False)["key"] for p in (1, 64)]
    assert keys == [autotune.workload_key([job], p) for p in (1, 64)]
    assert "wavefront" in autotune.KNOBS
    assert autotune.DEFAULT_GRID["queue_chunk"][0] == 64          # the kernel's default is timed first
