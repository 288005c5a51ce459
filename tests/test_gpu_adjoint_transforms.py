"""The adjoint's fixed-point transforms (csrc/adjoint_fix.cuh) against its FP64
Stockham ones, through the gradient: every class of line lengths along x and
along z, and odd lines along z, where a plane's last pair holds one line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (NX, NZ): lines of 3 NX/2 and 3 NZ/2 points
@pytest.mark.parametrize("nx,nz", [(240, 10), (384, 6), (200, 12), (10, 240), (6, 384), (8, 256), (160, 10), (12, 180),
                                   (32, 18), (48, 72)])
def test_fixed_point_and_stockham_gradients_agree(gpu_lib, nx, nz):
    """Each transform rounds by at most 3 eps log2(points) of its line, 1e-14, and
    the solves' own backward error is 2e-14; both pass through derivatives of norm
    1/dy^2 (2e3 on 17 points): 1e-10, and ten times that asserted.  A line left out
    or taken twice changes a gradient by its own size."""
    from owt.adjoint import seeded_wall_field
    from owt.ic import seeded_velocity
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.004, dkx=1.0, dkz=2.0, NX=nx, NY=17, NZ=nz, alpha_mesh=2.0, nu=1.0 / 3000.0)
    s = GpuSolver(p)
    s.init_fields(*seeded_velocity(p, seed=nx + nz))
    start = s.checkpoint()
    got = []
    for stockham in (False, True):
        s.use_stockham_fft(stockham)
        s.restore(start)
        s.set_wall_velocity(*[seeded_wall_field(p, q) for q in (1, 2)])
        got.append((s.drag_forward(3, 2),) + tuple(s.drag_backward()))
    s.close()
    for a, b in zip(*got):
        assert np.linalg.norm(b) > 0
        err = np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b)
        print(nx, nz, f"{err:.1e}")
        assert err < 1e-9
