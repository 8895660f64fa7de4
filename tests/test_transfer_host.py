"""The stress and the stress differential that the scatter and the Hessian product form from a
particle's HessianData (the left polar form), on the CPU, against the oracle's P and dP/dF: FP64
and the FP32 pairs, from light strain to inverted particles.

Tolerance, in rounding units times the scale of the terms: an entry of the stress is a sum of
four products of factors that carry two or three roundings each, about 16 in all; the
differential goes through three such products and a 3x3 inverse, about 64."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("transfer") / "transfer_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "non_ficks_diffusion_gb300", "csrc"),
                    "-I" + os.path.join(ROOT, "oracle"), "-x", "cu", os.path.join(HERE, "host", "transfer_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    return {k: float(v) for k, v in zip(out[::2], out[1::2])}


@pytest.mark.parametrize("family", ["light", "strained", "compressed", "stretched", "inverted"])
@pytest.mark.parametrize("bits", ["64", "32"])
def test_transfer_forms_match_the_oracle(check, family, bits):
    assert check["%s_P%s" % (family, bits)] <= 16
    assert check["%s_dP%s" % (family, bits)] <= 64
