"""owt_dy1_noalloc over the sizes it takes: its factors on the host for every NY
(tests/noalloc_block_check.cpp), and on the GPU the shortest lines, tiles of 64
lines with a remainder, tiles that shared memory limits, and in place, against
the handle's DY1 at the tolerance of the other routine tests (1e-12)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "open-3d-wallturbulence_gb300", "csrc")


def test_block_elimination_is_the_plain_one(tmp_path):
    exe = str(tmp_path / "noalloc_block_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + CSRC, os.path.join(ROOT, "tests", "noalloc_block_check.cpp"), "-o",
                    exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz", [(6, 7, 4), (250, 7, 250), (250, 32, 250), (20, 33, 18), (64, 257, 36), (64, 1025, 30)])
def test_sizes_and_in_place(gpu_lib, nx, ny, nz):
    import torch
    from owt import lib as L
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    lib = L.load(gpu_lib)
    p = CaseParams(dt=0.002, dkx=1.0, dkz=2.0, NX=nx, NY=ny, NZ=nz, alpha_mesh=2.0, nu=1e-3)
    rng = np.random.default_rng(ny)
    f = rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape)
    s = GpuSolver(p)
    want = s.dy(1, f)
    s.close()
    lines = p.NZ * p.NXH
    got = []
    for in_place in (False, True):
        a = torch.from_numpy(np.ascontiguousarray(np.transpose(f, (2, 0, 1)))).cuda()
        out = a if in_place else torch.full_like(a, float("nan"))
        rc = lib.owt_dy1_noalloc(ny, lines, 2.0, C.c_void_p(a.data_ptr()), C.c_void_p(out.data_ptr()),
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == L.OK, lib.owt_last_error(None).decode()
        torch.cuda.synchronize()
        got.append(np.transpose(out.cpu().numpy(), (1, 2, 0)))
    err = np.abs(got[0] - want).max() / np.abs(want).max()
    print(ny, lines, f"{err:.1e}")
    assert err < 1e-12
    np.testing.assert_array_equal(*got)
