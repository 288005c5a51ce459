"""FP64 transforms in 64-bit fixed point (csrc/transforms_fix.cuh): the Lamb
vector of six random spectral fields against numpy, beside the FP64 Stockham
kernels they replace, at the edges of the plan classes (lines of 6 to 576
points), with kx columns and (y, z) lines that do not fill a block.  Lengths
without a plan run the Stockham kernels in both arms, bitwise equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("velx", "vely", "velz", "vorx", "vory", "vorz")


def numpy_lamb(f, p):
    NZ, NZH, NXH, NX2, NZ2 = p.NZ, p.NZH, p.NXH, p.NX2, p.NZ2

    def phys(a):
        z = np.zeros((NZ2,) + a.shape[1:], complex)
        z[:NZH], z[NZ + 1:] = a[:NZH], a[NZH + 1:]
        x = np.zeros((NZ2, NX2 // 2 + 1, a.shape[2]), complex)
        x[:, :NXH] = np.fft.ifft(z, axis=0, norm="forward")
        return np.fft.irfft(x, n=NX2, axis=1, norm="forward")

    def spec(q):
        z = np.fft.fft(np.fft.rfft(q, axis=1, norm="forward")[:, :NXH], axis=0, norm="forward")
        return np.concatenate([z[:NZH], z[NZ:]], axis=0)

    u, v, w, ox, oy, oz = (phys(a) for a in f)
    return [spec(v * oz - w * oy), spec(w * ox - u * oz), spec(u * oy - v * ox)]


@pytest.mark.parametrize("nx,ny,nz", [(4, 7, 4), (6, 9, 10), (8, 7, 12), (30, 9, 20), (54, 7, 40), (96, 9, 64),
                                      (50, 7, 90), (108, 9, 128), (216, 7, 160), (200, 7, 216), (240, 9, 256),
                                      (288, 7, 320), (384, 7, 384), (320, 7, 24), (20, 7, 384), (250, 7, 300)])
def test_lamb_vector_matches_numpy(gpu_lib, nx, ny, nz):
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.002, dkx=1.0, dkz=2.0, NX=nx, NY=ny, NZ=nz, alpha_mesh=2.0, nu=1e-3)
    rng = np.random.default_rng(nx + nz)
    f = [rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape) for _ in FIELDS]
    for a in f:
        a[:, 0] = 0.0  # the library ignores the imaginary part of kx = 0 before the x transform only
    want = numpy_lamb(f, p)
    got = {}
    for arm in ("fixed", "stockham"):
        s = GpuSolver(p)
        s.use_stockham_fft(arm == "stockham")
        for n, a in zip(FIELDS, f):
            s.set(n, a)
        s.Lamb_vec()
        got[arm] = [s.get(n) for n in ("lmbx", "lmby", "lmbz")]
        s.close()
    # an FP64 transform of L points has a relative error of about eps log2 L;
    # two backward pairs enter the product, one forward pair follows
    tol = 3 * np.finfo(float).eps * np.log2(p.NX2 * p.NZ2)
    no_plan = {375, 450}
    for q in range(3):
        err = {a: np.linalg.norm(got[a][q] - want[q]) / np.linalg.norm(want[q]) for a in got}
        print(f"{nx}x{ny}x{nz} component {q}", {a: f"{e:.2e}" for a, e in err.items()}, f"tolerance {tol:.2e}")
        assert err["fixed"] < tol and err["stockham"] < tol
        if p.NX2 in no_plan and p.NZ2 in no_plan:
            assert np.array_equal(got["fixed"][q], got["stockham"][q])


def test_lines_that_are_not_finite_or_zero(gpu_lib):
    """A NaN reaches every mode of its y plane and no other plane; zero fields stay exactly zero."""
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.002, dkx=1.0, dkz=2.0, NX=32, NY=9, NZ=24, alpha_mesh=2.0, nu=1e-3)
    rng = np.random.default_rng(5)
    s = GpuSolver(p)
    s.Lamb_vec()
    assert all(np.array_equal(s.get(n), np.zeros(p.spectral_shape)) for n in ("lmbx", "lmby", "lmbz"))
    for n in FIELDS:
        a = rng.standard_normal(p.spectral_shape) + 1j * rng.standard_normal(p.spectral_shape)
        if n == "velx":
            a[3, 2, 4] = np.nan
        s.set(n, a)
    s.Lamb_vec()
    for n in ("lmby", "lmbz"):
        bad = ~np.isfinite(s.get(n))
        assert bad[:, :, 4].all() and not np.delete(bad, 4, axis=2).any()
    s.close()
