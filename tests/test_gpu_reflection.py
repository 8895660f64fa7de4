"""A body with inverted particles near a reflection, given by its initial Fe: one substep in each
precision against the oracle of that precision. The clamp brings the negative singular value
back to the lower limit, so that det Fe is positive again and Jp is about -1/0.975.

Tolerance of Jp: about 30 FP32 roundings of a quotient of products (64 of 2^-24), mixed one
rounding of the result (2), FP64 as its Jacobi SVD (1e-12). Fe moves by dt grad v Fe, and both
sides stop their CG at the same residual: velocities within 4 of it, gradients 64 (2/dx) times
that along each axis, and the FP32 rounding of entries near 1."""
import numpy as np
import pytest

import oracle_lib
from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp32", 64 * 2.0 ** -24), ("mixed", 2 * 2.0 ** -24), ("fp64", 1e-12)])
def test_inverted_particles_match_the_oracle(built_lib, prec, tol):
    desc, p = workloads.ball_scene(n=32, radius=0.1, velocity=(0.0, 0.0, 0.0), seed=4)
    n = len(p["mass"])
    rng = np.random.default_rng(4)
    q, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q *= np.sign(np.linalg.det(q))[:, None, None]
    s = np.array([1.004, 1.002, -0.996]) + 1e-3 * rng.random((n, 3))
    fe = (q * s[:, None, :]) @ np.transpose(q, (0, 2, 1))
    fe[::3] = np.eye(3)                      # among particles at rest
    p["Fe"] = fe.astype(np.float32).astype(np.float64).reshape(n, 9)
    ctx = capi.Context(precision=prec, max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.initialize()
    o = oracle_lib.oracle_from_desc(desc, p, precision=capi.PRECISIONS[prec])
    ctx.step(1e-6)
    o.step(1e-6)
    g, r = ctx.particles(0), o.particles()
    flipped = np.linalg.det(fe) < 0
    assert (r["Jp"][flipped] < -1.02).all()
    assert np.abs(g["Jp"] / r["Jp"] - 1).max() <= tol
    assert (np.linalg.det(g["Fe"][flipped]) > 0).all()
    assert np.abs(g["Fe"] - r["Fe"]).max() <= 1e-6 * 2 * 64 * 4 * o.stats()["cg_tolerance"] + 64 * 2.0 ** -24
    assert np.array_equal(g["valid"], r["valid"])
