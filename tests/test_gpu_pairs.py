"""The FP32 Hessian product's pair tables (two particles of one cell per lane) where they can
go wrong: lone particles, odd cells, a cell of one, two and many warps' worth of pairs, a
block of several work items, and few or many occupied cells per block. One substep whose CG
iterates against the FP32 oracle, in both forms of the product.

Tolerance: positions move by dt |v| < 1e-3, so their FP32 rounding is 2^-24 per unit; the two
sides stop the CG at the same relative tolerance 1e-5 of max|v*| < 10 m/s, so velocities may
differ by that tolerance times a few (4) iterations' worth of stopping slack."""
import numpy as np
import pytest

import oracle_lib
from non_ficks_diffusion_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

DT = 1e-4

CELLS = {
    "lone": [1],
    "odd": [1, 3, 5, 7, 9, 31, 33],
    "two_warps": [64, 65, 128, 1],
    "several_items": [1500, 700, 3],
    "full_block": [8] * 64,
    "ragged_block": [(5 * k) % 13 for k in range(64)],
}


def _scene(counts):
    desc, parts = workloads.ball_scene(n=32)
    rng = np.random.default_rng(len(counts))
    X = []
    for k, c in enumerate(counts):     # cells of the block at cells (12..15)^3
        cell = np.array([12 + k % 4, 12 + (k // 4) % 4, 12 + k // 16])
        X.append((cell + 0.05 + 0.9 * rng.random((c, 3))) / 32.0)
    X = np.concatenate(X).astype(np.float32).astype(np.float64)
    n = len(X)
    V = (rng.random((n, 3)) * 4 - 2).astype(np.float32).astype(np.float64)
    full = lambda a: np.full(n, np.float64(np.float32(a)))  # noqa: E731
    return desc, dict(X=X, V=V, mass=full(parts["mass"][0]), lambda0=full(parts["lambda0"][0]), mu0=full(parts["mu0"][0]))


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("cells", sorted(CELLS))
def test_pair_tables_match_the_oracle(built_lib, cells, form):
    desc, p = _scene(CELLS[cells])
    n = len(p["mass"])
    ctx = capi.Context(precision="fp32", max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.set_launch_config(hessian_warp_items=form)
    ctx.initialize()
    o = oracle_lib.oracle_from_desc(desc, p, precision=capi.FP32)
    ctx.step(DT)
    o.step(DT)
    g, r = ctx.particles(0), o.particles()
    assert n == 1 or o.stats()["cg_iterations"] > 0       # a lone particle starts converged
    assert np.abs(g["X"] - r["X"]).max() <= 4 * 2.0 ** -24 + 4 * 1e-5 * 10 * DT
    assert np.abs(g["V"] - r["V"]).max() <= 4 * 1e-5 * 10
