"""The mixed plasticity update against the FP64 one on the CPU, over yield limits (snow's, wide,
nearly and exactly a point, below and above 1, crossed) and singular values at, around, beyond
and on the negative side of them. Every sample counts, a NaN fails, and FP64 says which must yield.

Tolerances in units of 2^-24: rounding an exact result to FP32 is up to one unit for values just
above a power of two (Fe and Re over max(1, sy), Jp and Je relative), and a tenth is left for
the correction. The rotation of a particle that does not yield keeps the orthonormality of the FP32
one that it refines: 8 units (4 spacings, as for the whole update). The series' rotation and
det are exact results rounded: entries up to 1, Je up to 1.03, so one unit and a tenth."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "non_ficks_diffusion_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("clamp_limits") / "clamp_limits_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I" + CSRC, "-x", "cu", os.path.join(HERE, "host", "clamp_limits_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    return {k: float(v) for k, v in zip(out[::2], out[1::2])}


FAMILIES = ["mixed_sides", "lower", "upper", "pair", "spread", "inverted"]


@pytest.mark.parametrize("family", FAMILIES)
@pytest.mark.parametrize("limits", ["snow", "wide", "rigid", "point", "low", "high", "crossed"])
def test_mixed_clamp_rounds_like_fp64(check, limits, family):
    name = limits + "_" + family
    assert check[name + "_err"] <= 1.1
    assert check[name + "_rot"] <= 8
    # all singular values (5 % around the middle, or 10 % around 1) inside the band: none yields;
    # else a good part of the samples does
    if (limits, family) in (("wide", "mixed_sides"), ("wide", "pair"), ("low", "mixed_sides"), ("high", "mixed_sides")):
        assert check[name + "_yields"] == 0
    else:
        assert check[name + "_yields"] > 0.2


@pytest.mark.parametrize("strain,taken", [("rigid", 1.0), ("light", 1.0), ("limit", 0.3)])
def test_series_rounds_like_fp64(check, strain, taken):
    assert check["series_%s_taken" % strain] >= taken
    assert check["series_%s_err" % strain] <= 1.1
