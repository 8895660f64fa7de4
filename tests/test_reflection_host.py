"""Inverted particles near a reflection (det F < 0, F^T F near I) in FP32 and mixed storage, on
the CPU (mpm_math.cuh built as host code): such an F takes the SVD, whose negative singular value
the clamp brings back, in every precision.

Tolerances, u = 2^-24 the FP32 rounding unit. Je and Jp are products and quotients of a few
singular values: mixed rounds an FP64 result (2 u relative), FP32 makes about 30 roundings on
the way (64 u). Fe and Re: mixed rounds an FP64 result (entries up to 2: 2 u); the FP32 Jacobi's
vectors turn by its errors, some 16 u, over the gap of the singular values, at least 6e-4."""
import math
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "non_ficks_diffusion_gb300", "csrc")
U = 2.0 ** -24


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("reflection") / "reflection_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I" + CSRC, "-x", "cu", os.path.join(HERE, "host", "reflection_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    return {k: float(v) for k, v in zip(out[::2], out[1::2])}


@pytest.mark.parametrize("family", ["exact", "rigid", "light", "limit", "far"])
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_reflections_are_clamped_back(check, precision, family):
    name = precision + "_" + family
    assert check[name + "_det"] > 0.99
    assert check[name + "_scalars"] <= (2 if precision == "mixed" else 64) * U
    entries = check[name + "_entries"]
    assert not math.isnan(entries) and entries <= (2 * U if precision == "mixed" else 16 * U / 6e-4)
    assert check[name + "_rotations"] == 0
