"""The exponents the fixed-point FP64 transforms take, as the header states them:
fields scaled by powers of two give the same digits within the range, fields
below it count as zero, fields beyond it are not a number, and the Stockham
kernels take them all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IN = ("velx", "vely", "velz", "vorx", "vory", "vorz")
OUT = ("lmbx", "lmby", "lmbz")


def _lamb(s, fields, e):
    for n, f in zip(IN, fields):
        s.set(n, np.ldexp(f.real, e) + 1j * np.ldexp(f.imag, e))
    s.Lamb_vec()
    return [s.get(n) for n in OUT]


def _scaled(a, e):
    return np.ldexp(a.real, e) + 1j * np.ldexp(a.imag, e)


@pytest.mark.parametrize("nx,nz", [(32, 18), (96, 64), (240, 10)])
def test_range_of_the_lamb_vector(gpu_lib, nx, nz):
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.002, dkx=1.0, dkz=2.0, NX=nx, NY=7, NZ=nz, alpha_mesh=2.0, nu=1e-3)
    rng = np.random.default_rng(nx)
    fields = [rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape) for _ in IN]
    s = GpuSolver(p)
    one = _lamb(s, fields, 0)
    for e in (-450, -300, 300, 450):  # products of 2^-900 and 2^900 and their sums
        for a, b in zip(_lamb(s, fields, e), one):
            np.testing.assert_array_equal(a, _scaled(b, 2 * e))
    for e in (-900, -1000):  # every line below 2^-895
        assert not np.any(_lamb(s, fields, e))
    assert np.isnan(_lamb(s, fields, 1015)).all()
    s.use_stockham_fft(True)
    ref = _lamb(s, fields, 0)
    for e in (-450, 450):
        for a, b in zip(_lamb(s, fields, e), ref):
            np.testing.assert_array_equal(a, _scaled(b, 2 * e))
    s.close()


@pytest.mark.parametrize("e", [-900, 1008])
def test_stockham_takes_what_is_beyond(gpu_lib, e):
    """One field there and back: beyond the fixed-point range the option gives the
    field to FP64 rounding (3 eps log2 of the points, as its other tests)."""
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.002, dkx=1.0, dkz=2.0, NX=32, NY=7, NZ=18, alpha_mesh=2.0, nu=1e-3)
    rng = np.random.default_rng(1)
    f = rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape)
    f[p.NZH] = 0
    f[:, 0] = 0
    s = GpuSolver(p)
    s.use_stockham_fft(True)
    back = s.Physical2Fourier_dealiased(s.Fourier2Physical_dealiased(_scaled(f, e)))
    s.close()
    err = np.linalg.norm(_scaled(back, -e) - f) / np.linalg.norm(f)
    assert err < 6 * np.finfo(float).eps * np.log2(p.NX2 * p.NZ2)
