"""A small scene whose cooperative solve is refused (a stand-in in the library answers for the launch)
steps with the loop of kernels: the same substeps and frames as with MPM_COOP=0, which never asks
for it, and the launches of the loop.

Tolerance: both run the same kernels, and their FP32 sums differ in order only. Both stop at a
residual of 1e-5 max|v*|, so a velocity may differ by that tolerance times a few (4) when one
stops an iteration earlier, a position by dt times that."""
import numpy as np
import pytest

from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

DT = 1e-4


def _run(monkeypatch, coop, frames):
    monkeypatch.setenv("MPM_COOP", coop)
    desc, p = workloads.ball_scene(n=32, center=(0.5, 0.2, 0.5), radius=0.1, velocity=(1.0, -4.0, 0.5), seed=5)
    ctx = capi.Context(precision="fp32", max_particles=len(p["mass"]), max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.initialize()
    before = ctx.stats(0)["gpu_launches"]
    steps = ctx.advance_to_time(4 * DT) if frames else 4
    if not frames:
        ctx.step(DT, 2)
        ctx.step(DT, 2)
    s = ctx.stats(0)
    return ctx.particles(0), steps, s["gpu_launches"] - before


@pytest.mark.parametrize("frames", [False, True])
def test_refused_solve_runs_the_loop(built_lib, monkeypatch, frames):
    a, na, la = _run(monkeypatch, "refuse", frames)
    b, nb, lb = _run(monkeypatch, "0", frames)
    c, nc, lc = _run(monkeypatch, "1", frames)
    assert na == nb == nc
    assert abs(la - lb) <= 2 * 4 * na and lc < la      # an iteration (two kernels) more or less in a substep
    tol = 4 * 1e-5 * 5.0
    for k in (b, c):
        assert np.abs(a["V"] - k["V"]).max() <= tol * na
        assert np.abs(a["X"] - k["X"]).max() <= tol * na * na * 5e-3 + 4 * 2.0 ** -24
