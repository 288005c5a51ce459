"""The per-line kernels whose operator tables live in shared memory, on both
sides of the lengths where the tables no longer fit and are read from device
memory: the nonlinear source (from 2322 wall-normal points), DY2 of uploaded
histories, and the adjoint's nonlinear source (1862) and mean mode (510)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(ny, **kw):
    from owt.params import CaseParams
    return CaseParams(**{**dict(dt=1e-4, dkx=1.0, dkz=2.0, NX=6, NY=ny, NZ=4, alpha_mesh=2.0, nu=1e-3), **kw})


@pytest.mark.parametrize("ny", [7, 8, 257, 2321, 2322, 2401])
def test_nonlinear_source_is_its_formula(gpu_lib, ny):
    """Hg = i kz lx - i kx lz and Hv = -k^2 ly - DY1 (i kx lx + i kz lz) with the
    start-up kernel's DY1: both apply the same well-conditioned A1, so they agree
    to some tens of roundings of the largest value: 200 eps."""
    from owt.solver import GpuSolver
    p = _params(ny)
    s = GpuSolver(p)
    rng = np.random.default_rng(ny)
    lx, ly, lz = (rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape) for _ in range(3))
    for n, a in zip(("lmbx", "lmby", "lmbz"), (lx, ly, lz)):
        s.set(n, a)
    s.nonlinear_source()
    kx = (p.dkx * np.arange(p.NXH))[None, :, None]
    kz = (p.dkz * np.array([k if k < p.NZH else k - p.NZ for k in range(p.NZ)]))[:, None, None]
    hg = 1j * kz * lx - 1j * kx * lz
    hv = -(kx ** 2 + kz ** 2) * ly - s.dy(1, 1j * kx * lx + 1j * kz * lz)
    for n, want in (("Hg", hg), ("Hv", hv)):
        err = np.abs(s.get(n) - want).max() / np.abs(want).max()
        print(ny, n, f"{err:.1e}")
        assert err < 200 * np.finfo(float).eps
    s.close()


@pytest.mark.parametrize("ny", [65, 1900])
def test_uploaded_history_gives_the_resident_step(gpu_lib, ny):
    """DY2 v re-derived from uploaded levels against the solves' own: a solve's
    backward error 2e-14 through an operator of norm 1/dy^2 (1e7 on the longer
    grid) is 2e-7 of v's second derivative; 1e-5 of the field asserted."""
    from owt.ic import seeded_velocity
    from owt.solver import GpuSolver
    p = _params(ny)
    got = []
    for upload in (False, True):
        s = GpuSolver(p)
        s.init_fields(*seeded_velocity(p, seed=3))
        s.time_Integration(3)
        if upload:
            for n in ("vely_0", "vely_1", "vely_2"):
                s.set(n, s.get(n))
        s.time_Integration(1)
        got.append(s.get("vely"))
        s.close()
    assert np.linalg.norm(got[1] - got[0]) < 1e-5 * np.linalg.norm(got[0])


@pytest.mark.parametrize("ny", [509, 510, 1901])
def test_drag_gradient_is_its_central_difference(gpu_lib, ny):
    """Three steps of wall blowing, one seeded direction.  A step's mean force is
    quadratic in the fields of the step before, and the fields are linear in the
    wall velocity and in the sources, which are quadratic in the fields before:
    after three steps the drag is a polynomial of degree four, for which the
    five-point difference is exact.  The bound is that of the Re_tau=180
    comparison, 1e-5."""
    from owt.adjoint import seeded_wall_field
    from owt.ic import seeded_velocity
    from owt.solver import GpuSolver
    p = _params(ny)
    s = GpuSolver(p)
    s.init_fields(*seeded_velocity(p, seed=2))
    start = s.checkpoint()
    wall = [seeded_wall_field(p, q) for q in (1, 2)]
    d = [seeded_wall_field(p, q, 1.0) for q in (101, 102)]
    s.set_wall_velocity(*wall)
    s.drag_forward(3, 2)
    grad = s.drag_backward()
    eps, J = 1e-3, []
    for k in (1, -1, 2, -2):
        s.restore(start)
        s.set_wall_velocity(*(w + k * eps * q for w, q in zip(wall, d)))
        J.append(s.drag_forward(3, 3))
    fd = (8 * (J[0] - J[1]) - (J[2] - J[3])) / (12 * eps)
    ad = float(sum(np.real(np.vdot(g, q)) for g, q in zip(grad, d)))
    print(ny, f"adjoint {ad:.8e} difference {fd:.8e}")
    assert abs(fd - ad) <= 1e-5 * abs(ad)
    s.close()
