"""Wall-normal statistics of a state that is not finite say so: a NaN in a mean
or in a fluctuation of one y plane makes the RMS of that component there NaN,
and leaves the other planes and components as they were."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [(0, 0), (3, 2), (5, 0)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("name,rms", [("velx", "u_rms"), ("vely", "v_rms"), ("velz", "w_rms")])
def test_not_finite_shows_in_its_plane(gpu_lib, mode, value, name, rms):
    from owt.ic import seeded_velocity
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.004, dkx=1.0, dkz=2.0, NX=16, NY=17, NZ=12, alpha_mesh=2.0, nu=1.0 / 3000.0)
    s = GpuSolver(p)
    fields = dict(zip(("velx", "vely", "velz"), seeded_velocity(p, seed=1)))
    for n, f in fields.items():
        s.set(n, f)
    good = s.statistics()
    f = fields[name].copy()
    f[mode][6] = value
    s.set(name, f)
    got = s.statistics()
    s.close()
    assert np.isfinite([good[n] for n in GpuSolver.STAT_NAMES]).all()
    assert not np.isfinite(got[rms][6])
    others = {"velx": ("v_rms", "w_rms"), "vely": ("u_rms", "w_rms"), "velz": ("u_rms", "v_rms", "uv")}[name]
    for n in others:
        np.testing.assert_array_equal(got[n], good[n])
    np.testing.assert_array_equal(np.delete(got[rms], 6), np.delete(good[rms], 6))
