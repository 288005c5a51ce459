"""The mode kernel's adjoint on packed factor streams (csrc/adjoint_modes.cu):
the objective and the gradient of the full-band solves, bit for bit (the streams
leave out exact zeros only), for wall-normal sizes without an interior, with few
interior columns and with columns left over (odd NY), modes that do not fill the
last group of 16, and both orders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,order", [(4, 7, 4, 8), (12, 9, 10, 8), (16, 17, 16, 8), (10, 18, 12, 8),
                                            (18, 19, 8, 8), (20, 20, 24, 8), (24, 33, 18, 8), (36, 34, 10, 8),
                                            (40, 98, 36, 8), (16, 17, 16, 6), (20, 33, 24, 6), (32, 66, 20, 6)])
def test_streams_give_the_full_band_gradient(gpu_lib, nx, ny, nz, order):
    from owt.adjoint import seeded_wall_field
    from owt.ic import seeded_velocity
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.004, dkx=1.0, dkz=2.0, NX=nx, NY=ny, NZ=nz, alpha_mesh=2.0, nu=1.0 / 3000.0, fd_order=order)
    got = []
    for dense in (False, True):
        s = GpuSolver(p)
        s.force_dense_bands(dense)
        s.init_fields(*seeded_velocity(p, seed=ny))
        s.set_wall_velocity(*[seeded_wall_field(p, q) for q in (1, 2)])
        got.append((s.drag_forward(3, 2),) + tuple(s.drag_backward()))
        s.close()
    assert np.abs(got[0][1]).max() > 0
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
