"""The one-kernel CG solve of a small single scene against the loop of kernels that larger scenes
and batches run (hessian_warp_items = 0 selects it): from one work item to more work items
than resident CTAs, snow and fluid, barrier contact, iteration limits, frames.

Tolerance: both stop at a residual of 1e-5 max|v*| and differ in the order of FP32 sums only,
so a velocity may differ by that tolerance times a few (4) when one stops an iteration
earlier, a position by dt times that."""
import numpy as np
import pytest

from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

DT = 1e-4


def _run(desc, p, precision, form, step, density=None):
    n = len(p["mass"])
    ctx = capi.Context(precision=precision, max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, Jp=None if density is None else np.full(n, density), **p)
    ctx.set_launch_config(hessian_warp_items=form)
    ctx.initialize()
    status = step(ctx)
    return ctx.particles(0), ctx.stats(0), status


def _same(a, b, vmax, steps):
    (pa, sa, ra), (pb, sb, rb) = a, b
    assert ra == rb and sa["cg_converged"] == sb["cg_converged"]
    assert abs(sa["cg_iterations"] - sb["cg_iterations"]) <= 1
    assert np.array_equal(pa["valid"], pb["valid"])
    tol = 4 * 1e-5 * vmax
    assert np.abs(pa["V"] - pb["V"]).max() <= tol * steps
    assert np.abs(pa["X"] - pb["X"]).max() <= tol * steps * steps * DT + 4 * 2.0 ** -24
    return sa


# particles per body: 8 (one work item) to 800K (more work items than the CTAs that fit the GPU)
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("n,radius", [(16, 0.07), (32, 0.1), (48, 0.25), (64, 0.25), (96, 0.3)])
def test_one_kernel_solve_matches_the_loop(built_lib, precision, n, radius):
    desc, p = workloads.ball_scene(n=n, center=(0.5, radius + 2.2 / n, 0.5), radius=radius, velocity=(1.0, -6.0, 0.0), seed=n)
    rng = np.random.default_rng(n)
    p["V"] = p["V"] + rng.random(p["V"].shape) * 2 - 1
    runs = [_run(desc, p, precision, form, lambda c: c.step(DT, 3)) for form in (2, 0)]
    assert _same(runs[0], runs[1], 8.0, 3)["cg_iterations"] > 0


def test_one_kernel_solve_of_a_fluid(built_lib):
    desc, p = workloads.ball_scene(n=32, radius=0.15, velocity=(0.0, -1.0, 0.0), density=2.0, seed=3)
    desc.material, desc.bulk_modulus, desc.eos_gamma, desc.plastic = capi.MATERIAL_EOS_FLUID, 1.0, 7.0, 0
    runs = [_run(desc, p, "fp32", form, lambda c: c.step(DT, 3), density=2.0) for form in (2, 0)]
    _same(runs[0], runs[1], 2.0, 3)


@pytest.mark.parametrize("most,least", [(0, 0), (1, 0), (50, 5)])
def test_one_kernel_solve_keeps_the_iteration_limits(built_lib, most, least):
    desc, p = workloads.ball_scene(n=32, center=(0.5, 0.17, 0.5), radius=0.1, velocity=(0.0, -16.0, 0.0), seed=31)
    desc.cg_max_iters, desc.cg_min_iters = most, least
    runs = [_run(desc, p, "fp32", form, lambda c: c.step(DT, 1)) for form in (2, 0)]
    st = _same(runs[0], runs[1], 17.0, 1)
    # the solver also stops before cg_min_iters once the residual is below the FP32 epsilon
    assert st["cg_iterations"] >= least or st["cg_residual"] < 2.0 ** -23
    assert most > 1 or st["cg_iterations"] == most
    assert runs[0][2] == (capi.OK if most > 1 else capi.CG_NOT_CONVERGED)


def test_frames_with_the_one_kernel_solve(built_lib):
    desc, p = workloads.ball_scene(n=32, center=(0.5, 0.2, 0.5), radius=0.1, velocity=(1.0, -4.0, 0.5), seed=5)
    runs = [_run(desc, p, "mixed", form, lambda c: c.advance_to_time(0.005)) for form in (2, 0)]
    assert runs[0][2] > 1
    _same(runs[0], runs[1], 5.0, runs[0][2])
