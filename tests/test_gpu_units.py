"""Units of work items (128 pairs each, one pass for each warp of a CTA), by which the FP32
scatter, the one-kernel CG solve and G2P are dealt out: work items just below, at and above one
and several units, items of lone particles (more pairs than half the particles), and a block
of two work items, beside a resting cube of 4,096 particles (fewer are not dealt out). One
substep in the default form against the FP32 oracle.

Tolerance: as in the pair-table test. Positions move by dt |v| < 1e-3, so their FP32 rounding is
2^-24 per unit; both sides stop the CG at 1e-5 of max|v*| < 10 m/s, so velocities may differ
by that times a few (4) iterations' worth of stopping slack."""
import numpy as np
import pytest

import oracle_lib
from non_ficks_diffusion_gb300 import capi
from test_gpu_pairs import DT, _scene

pytestmark = pytest.mark.gpu

CELLS = {
    "255": [255], "256": [256], "257": [257], "512": [512], "513": [513],
    "64_lone": [1] * 64, "128_pairs": [3] * 64, "192_pairs": [5] * 64,
    "full_item": [16] * 64, "item_and_one": [16] * 63 + [17],
}


@pytest.mark.parametrize("cells", sorted(CELLS))
def test_units_match_the_oracle(built_lib, cells):
    desc, p = _scene(CELLS[cells])
    rng = np.random.default_rng(7)
    cell = np.stack(np.meshgrid(*[np.arange(20, 28)] * 3, indexing="ij"), -1).reshape(-1, 3).repeat(8, 0)
    X = ((cell + 0.05 + 0.9 * rng.random((4096, 3))) / 32.0).astype(np.float32).astype(np.float64)
    rest = {"X": X, "V": np.zeros((4096, 3)), **{k: np.full(4096, p[k][0]) for k in ("mass", "lambda0", "mu0")}}
    p = {k: np.concatenate([p[k], rest[k]]) for k in p}
    n = len(p["mass"])
    ctx = capi.Context(precision="fp32", max_particles=n, max_scenes=1)
    ctx.add_scene(desc)
    ctx.add_particles(0, **p)
    ctx.initialize()
    o = oracle_lib.oracle_from_desc(desc, p, precision=capi.FP32)
    ctx.step(DT)
    o.step(DT)
    g, r = ctx.particles(0), o.particles()
    assert o.stats()["cg_iterations"] > 0
    assert np.abs(g["X"] - r["X"]).max() <= 4 * 2.0 ** -24 + 4 * 1e-5 * 10 * DT
    assert np.abs(g["V"] - r["V"]).max() <= 4 * 1e-5 * 10
