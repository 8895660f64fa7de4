"""The mixed plasticity update's FP32 correction of the SVD against the FP64 clamp, on the CPU
(the kernels' mpm_math.cuh built as host code). Rounding an exact result to FP32 is an error
of up to one unit of 2^-24 (entries up to 2, Jp and Je relative to a value just above a power
of two); a tenth of a unit is left for the correction itself."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "non_ficks_diffusion_gb300", "csrc")


@pytest.fixture(scope="module")
def clamp_check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("clamp") / "clamp_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I" + CSRC, "-x", "cu", os.path.join(HERE, "host", "clamp_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    return {k: float(v) for k, v in zip(out[::2], out[1::2])}


@pytest.mark.parametrize("family", ["wide", "band", "equal", "lower", "upper", "near", "pair", "far"])
def test_corrected_clamp_rounds_like_fp64(clamp_check, family):
    assert clamp_check[family] <= 1.1


@pytest.mark.parametrize("family", ["rigid", "light", "limit"])
def test_rotation_near_a_rotation_rounds_like_fp64(clamp_check, family):
    # entries up to 1: half a unit of rounding, and a tenth for the series' end
    assert clamp_check[family] <= 0.6
