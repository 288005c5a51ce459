"""A reverse sweep whose tape does not fit the device is refused, and the handle
goes on: the next gradient is the one from before, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_refused_tape_leaves_the_gradient_as_it_was(gpu_lib):
    from owt.adjoint import seeded_wall_field
    from owt.ic import seeded_velocity
    from owt.lib import OwtError
    from owt.params import CaseParams
    from owt.solver import GpuSolver
    p = CaseParams(dt=0.004, dkx=1.0, dkz=2.0, NX=12, NY=17, NZ=8, alpha_mesh=2.0, nu=1.0 / 3000.0)
    s = GpuSolver(p)
    s.init_fields(*seeded_velocity(p, seed=5))
    start = s.checkpoint()

    def gradient(steps, interval):
        s.restore(start)
        s.set_wall_velocity(*[seeded_wall_field(p, q) for q in (1, 2)])
        return (s.drag_forward(steps, interval),) + tuple(s.drag_backward())

    want = gradient(3, 2)
    with pytest.raises(OwtError) as e:
        gradient(1, 10 ** 9)  # a tape of 78 TB: the allocation fails at once
    assert e.value.code == 5
    for a, b in zip(gradient(3, 2), want):
        np.testing.assert_array_equal(a, b)
    s.close()
