"""An upper yield limit below -1 (crossed with the lower one), FP32 and mixed storage against FP64 on
the CPU: an F near a rotation is not inside such a band, though the limit's square exceeds 1.

Tolerances in units of 2^-24: mixed rounds an exact result (one unit) with a tenth
for the correction; FP32 makes some 30 roundings on the way to Je and Jp, and its Jacobi's
factors are orthonormal to about 16 units, twice in a product: 64."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "non_ficks_diffusion_gb300", "csrc")


def test_upper_limit_below_minus_one(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "negative_yield_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I" + CSRC, "-x", "cu", os.path.join(HERE, "host", "negative_yield_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    err = {k: float(v) for k, v in zip(out[::2], out[1::2])}
    for q in ("entries", "scalars"):
        assert err["mixed_" + q] <= 1.1
        assert err["fp32_" + q] <= 64
