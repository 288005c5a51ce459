"""The first and second derivatives' stencil rows as the kernels read them
(csrc/setup_host.cpp, stencil_rows; tests/stencil_rows_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "open-3d-wallturbulence_gb300", "csrc")


def test_rows_keep_their_places(tmp_path):
    exe = str(tmp_path / "stencil_rows_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + CSRC, os.path.join(ROOT, "tests", "stencil_rows_check.cpp"),
                    os.path.join(CSRC, "setup_host.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
