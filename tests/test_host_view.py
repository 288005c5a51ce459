"""Host arrays that kernels write or read directly (csrc/host_view.h) lie as a
whole in one page-locked range with that access; all others are staged
(tests/host_view_check.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "open-3d-wallturbulence_gb300", "csrc")


def _run(tmp_path, *args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc absent")
    exe = str(tmp_path / "host_view_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I" + CSRC, os.path.join(ROOT, "tests", "host_view_check.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_rule_takes_whole_ranges_only(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_real_allocations_and_registrations(tmp_path):
    _run(tmp_path, "gpu")
