"""Solver limits at the ends of what a scene may ask for, in the one-kernel CG solve and in the loop
of kernels: tolerances below zero (the iterations run to their limit)
and an iteration limit of 2^31 - 1 (it runs to convergence, as a smaller one that suffices)."""
import pytest

from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

DT = 1e-4


def _scene(**kw):
    desc, p = workloads.ball_scene(n=32, center=(0.5, 0.17, 0.5), radius=0.1, velocity=(0.0, -16.0, 0.0), seed=31)
    for k, v in kw.items():
        setattr(desc, k, v)
    return desc, p


def _step(desc, p, precision, form, graphs=True):
    ctx = capi.Context(precision=precision, max_particles=len(p["mass"]), max_scenes=1, use_graphs=graphs)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.set_launch_config(hessian_warp_items=form)
    ctx.initialize()
    status = ctx.step(DT)
    return status, ctx.stats(0)


@pytest.mark.parametrize("form", [2, 0])
@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
def test_negative_tolerance_runs_to_the_limit(built_lib, precision, form):
    status, s = _step(*_scene(cg_abs_tol=-1.0, cg_rel_tol=-1.0, cg_max_iters=5), precision, form)
    assert status == capi.CG_NOT_CONVERGED
    assert s["cg_iterations"] == 5 and not s["cg_converged"] and s["cg_tolerance"] < 0


@pytest.mark.parametrize("form,graphs", [(2, True), (0, True), (0, False)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_largest_iteration_limit(built_lib, precision, form, graphs):
    status, s = _step(*_scene(cg_max_iters=2 ** 31 - 1), precision, form, graphs)
    expected, e = _step(*_scene(cg_max_iters=1000), precision, form, graphs)
    assert status == expected == capi.OK and e["cg_iterations"] > 1
    assert s["cg_converged"] and abs(s["cg_iterations"] - e["cg_iterations"]) <= 1
