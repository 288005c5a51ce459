"""The mode kernel on packed factor streams (csrc/modes_stream.cuh): the same
bits as the pair mapping after three steps with wall blowing, for wall-normal
sizes without an interior, with one quad of interior columns and with two
columns left over in the omega_y-system (odd NY), and modes that do not fill
the last group of 16; the sixth-order option against its full-band solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("vely", "vory", "velx", "velz", "vorx", "vorz", "Hv", "Hg")


def run(s, vel, wall):
    s.init_fields(*vel)
    s.set_wall_velocity(*wall)
    s.time_Integration(3)
    return [s.get(n) for n in NAMES]


def case(nx, ny, nz, order):
    from owt.adjoint import seeded_wall_field
    from owt.ic import seeded_velocity
    from owt.params import CaseParams
    p = CaseParams(dt=0.004, dkx=1.0, dkz=2.0, NX=nx, NY=ny, NZ=nz, alpha_mesh=2.0, nu=1.0 / 3000.0, fd_order=order)
    return p, seeded_velocity(p, seed=ny), [seeded_wall_field(p, q) for q in (1, 2)]


@pytest.mark.parametrize("nx,ny,nz", [(4, 7, 4), (12, 9, 10), (16, 17, 16), (10, 18, 12), (18, 19, 8), (20, 20, 24),
                                      (24, 33, 18), (36, 34, 10), (32, 65, 32), (40, 98, 36)])
def test_streams_give_the_pair_mapping_bits(gpu_lib, nx, ny, nz):
    from owt.solver import GpuSolver
    p, vel, wall = case(nx, ny, nz, 8)
    s = GpuSolver(p)
    s.force_modes_variant(0)
    want = run(s, vel, wall)
    if not s.info("sparse_solve"):
        pytest.skip("full-band solve at this size")
    n = s.info("modes_variants")
    for var in (n - 2, n - 1):
        s.force_modes_variant(var)
        for name, a, b in zip(NAMES, run(s, vel, wall), want):
            np.testing.assert_array_equal(a, b, err_msg=f"variant {var}: {name}")
    s.close()


@pytest.mark.parametrize("nx,ny,nz", [(16, 17, 16), (20, 33, 24), (32, 66, 20)])
def test_sixth_order_streams_give_the_full_band_bits(gpu_lib, nx, ny, nz):
    from owt.solver import GpuSolver
    p, vel, wall = case(nx, ny, nz, 6)
    got = []
    for dense in (False, True):
        s = GpuSolver(p)
        s.force_dense_bands(dense)
        got.append(run(s, vel, wall))
        s.close()
    for name, a, b in zip(NAMES, *got):
        np.testing.assert_array_equal(a, b, err_msg=name)
