"""The CG of a material so stiff and so fast that s^T K s itself leaves FP32 (about 1e45 at the body's edge) while
dt^2 s^T K s is small beside the masses: one substep against the oracle in every form of the
Hessian product. The step is 1e-14 so that particles stay where they are.

Tolerance: both sides stop their CG at the same residual, so velocities may differ by that times
a few (4) iterations' worth of stopping slack."""
import numpy as np
import pytest

import oracle_lib
from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [2, 0, 1])
@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
def test_stiff_and_fast_snow(built_lib, prec, form):
    desc, p = workloads.ball_scene(n=16, radius=0.2, velocity=(0.0, 0.0, 0.0), seed=6)
    n = len(p["mass"])
    p["V"] = 1e10 * (2 * np.random.default_rng(6).random((n, 3)) - 1)
    p["lambda0"], p["mu0"] = 1e21 * p["lambda0"], 1e21 * p["mu0"]
    ctx = capi.Context(precision=prec, max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.set_launch_config(hessian_warp_items=form)
    ctx.initialize()
    o = oracle_lib.oracle_from_desc(desc, p, precision=capi.PRECISIONS[prec])
    st = ctx.step(1e-14)
    o.step(1e-14)
    g, r, so = ctx.particles(0), o.particles(), o.stats()
    assert so["converged"] and so["cg_iterations"] > 0 and np.isfinite(r["V"]).all()
    assert st == capi.OK
    assert np.array_equal(g["valid"], r["valid"])
    assert np.abs(g["V"] - r["V"]).max() <= 4 * so["cg_tolerance"]
