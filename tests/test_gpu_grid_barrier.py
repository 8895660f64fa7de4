"""The grid barrier of the one-kernel CG solve on its own: its count of arrivals wraps (from just
below 2^32) without letting a CTA through early, and with a CTA that never arrives the others give
up after their limit, the call reports it, and the context goes on stepping."""
import numpy as np
import pytest

from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def _ctx():
    desc, parts = workloads.ball_scene(n=32, radius=0.12)
    ctx = capi.Context(precision="fp32", max_particles=len(parts["mass"]), max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **parts)
    ctx.initialize()
    return ctx


# first arrivals before 2^32: none, in the middle of a barrier's arrivals, at a barrier's end
# (152 CTAs), at half the range
@pytest.mark.parametrize("first", [0, 2 ** 32 - 1, 2 ** 32 - 700, 2 ** 32 - 152, 2 ** 31 - 5])
def test_arrivals_wrap(built_lib, first):
    ctx = _ctx()
    for phases in (1, 64):
        assert ctx.L.mpm_selftest_grid_barrier(ctx.h, first, phases, 0, 1 << 20) == capi.OK


@pytest.mark.parametrize("spin_limit", [1, 1000, 20000])
def test_grid_wait_gives_up_and_reports(built_lib, spin_limit):
    ctx = _ctx()
    before = ctx.particles(0)
    assert ctx.L.mpm_selftest_grid_barrier(ctx.h, 0, 2, 1, spin_limit) == capi.CUDA_ERROR
    assert b"CG grid barrier wait exceeded its limit" in ctx.L.mpm_last_error(ctx.h)
    assert ctx.L.mpm_selftest_grid_barrier(ctx.h, 0, 0, 0, 1000) == capi.BAD_ARG
    assert ctx.L.mpm_selftest_grid_barrier(ctx.h, 0, 65, 0, 1000) == capi.BAD_ARG
    assert ctx.L.mpm_selftest_grid_barrier(ctx.h, 0, 1, 0, (1 << 20) + 1) == capi.BAD_ARG
    assert np.array_equal(before["X"], ctx.particles(0)["X"])
    assert ctx.step(1e-4, 2) == capi.OK
    assert np.isfinite(ctx.particles(0)["X"]).all()
