"""The fixed-point line transforms of the FP64 transform kernels
(csrc/fft_fix.cuh), compiled by nvcc as host code and checked against a direct
transform in long double (tests/fft_fix_check.cu): every length with a plan,
both signs, an error no larger than an FP64 transform's, and the ends of the
range."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "open-3d-wallturbulence_gb300", "csrc")


def test_fixed_point_transforms_match_direct_dft(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc absent")
    exe = str(tmp_path / "fft_fix_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-w", "-I" + CSRC, os.path.join(ROOT, "tests", "fft_fix_check.cu"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
