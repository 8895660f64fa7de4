"""A fluid in SI units: water, 1000 kg/m^3, bulk modulus 2.2e9 and exponent 7, whose pressure
coefficient V0/rho k rho^(gamma-1) is 6.6e19 on a 16^3 grid, too large for the powers that the 3x3
system of snow's stress takes. One substep in FP32 storage against the oracle, in every form of
the Hessian product; a time step of 1e-15 keeps speeds (about 1e8) and positions in range.

Tolerance: both sides stop their CG at the same residual, 1e-5 of the largest grid speed, so
velocities may differ by that times a few (4) iterations' worth of stopping slack; the rounding
of the forces (sums of about 64 cancelling terms) is a hundredth of it."""
import numpy as np
import pytest

import oracle_lib
from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [2, 0, 1])
@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
def test_water_in_si_units(built_lib, prec, form):
    desc, p = workloads.ball_scene(n=16, radius=0.2, velocity=(0.0, -1.0, 0.0), density=1000.0, seed=3)
    desc.material, desc.bulk_modulus, desc.eos_gamma, desc.plastic = capi.MATERIAL_EOS_FLUID, 2.2e9, 7.0, 0
    n = len(p["mass"])
    p["Jp"] = np.full(n, 1000.0)
    ctx = capi.Context(precision=prec, max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.set_launch_config(hessian_warp_items=form)
    ctx.initialize()
    o = oracle_lib.oracle_from_desc(desc, p, precision=capi.PRECISIONS[prec])
    assert ctx.step(1e-15) == capi.OK
    o.step(1e-15)
    g, r = ctx.particles(0), o.particles()
    vmax = np.abs(r["V"]).max()
    assert np.isfinite(r["V"]).all() and vmax > 1e4
    assert np.array_equal(g["valid"], r["valid"])
    assert np.abs(g["V"] - r["V"]).max() <= 4 * o.stats()["cg_tolerance"]
