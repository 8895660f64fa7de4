"""The grid barrier of the one-kernel CG solve on its own: its count of arrivals wraps (from just
below 2^32) without letting a CTA through early."""
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
