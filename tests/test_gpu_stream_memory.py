"""The packed factor streams are a second copy of the factors: where they do not
fit (a limit stands for the device's end), whole or after a few of their parts,
steps, gradients, host-state steps and batches run on the band storage with the
same bits, nothing of them stays allocated, and they come back when there is
room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("velx", "vely", "velz", "vorx", "vory", "vorz", "Hv", "Hg")


def _params(order, **kw):
    from owt.params import CaseParams
    return CaseParams(**{**dict(dt=0.004, dkx=1.0, dkz=2.0, NX=20, NY=33, NZ=24, alpha_mesh=2.0, nu=1.0 / 3000.0,
                                fd_order=order), **kw})


def _solver(p, seed=3):
    from owt.ic import seeded_velocity
    from owt.solver import GpuSolver
    s = GpuSolver(p)
    s.use_graph(True)
    s.init_fields(*seeded_velocity(p, seed=seed))
    return s


def _same(a, b):
    for n in FIELDS:
        np.testing.assert_array_equal(a.get(n), b.get(n), err_msg=n)


@pytest.fixture(scope="module", params=[8, 6])
def reference(request, gpu_lib):
    """A channel that has its streams, after three steps, and what they hold."""
    s = _solver(_params(request.param))
    before = s.info("device_bytes")
    s.time_Integration(3)
    yield request.param, s, s.info("device_bytes") - before
    s.close()


@pytest.mark.parametrize("share", [0.0, 0.4, 0.999])
def test_steps_without_room_for_the_streams(reference, share):
    order, ref, size = reference
    assert size > 0
    s = _solver(_params(order))
    before = s.info("device_bytes")
    s.limit_stream_bytes(int(share * size))
    for _ in range(3):
        s.time_Integration(1)
        assert s.info("device_bytes") == before
    assert "stream" not in s.tuning_report()
    _same(s, ref)
    s.limit_stream_bytes(-1)
    s.limit_stream_bytes(size)  # exactly enough
    s.time_Integration(1)
    assert s.info("device_bytes") == before + size
    s.close()


def test_streams_taken_away_between_steps(reference):
    order, ref, size = reference
    s = _solver(_params(order))
    s.time_Integration(1)
    held = s.info("device_bytes")
    s.limit_stream_bytes(0)
    assert s.info("device_bytes") == held - size
    s.time_Integration(1)
    s.limit_stream_bytes(-1)
    s.time_Integration(1)
    assert s.info("device_bytes") == held
    _same(s, ref)
    s.close()


def test_gradient_without_the_streams_and_after_they_were_given_back(reference):
    from owt.adjoint import seeded_wall_field
    from owt.lib import OwtError
    order, _, size = reference
    got = []
    for limit in (-1, 0):
        s = _solver(_params(order))
        s.limit_stream_bytes(limit)
        start = s.checkpoint()

        def gradient(steps, interval):
            s.restore(start)
            s.set_wall_velocity(*[seeded_wall_field(s.params, q) for q in (1, 2)])
            return (s.drag_forward(steps, interval),) + tuple(s.drag_backward())

        got.append(gradient(3, 2))
        held = s.info("device_bytes")
        with pytest.raises(OwtError) as e:
            gradient(1, 10 ** 9)  # no device has room for this tape
        assert e.value.code == 5
        assert s.info("device_bytes") == held - (size if limit else 0)
        got.append(gradient(3, 2))
        assert s.info("device_bytes") == held
        s.close()
    for g in got[1:]:
        for a, b in zip(g, got[0]):
            np.testing.assert_array_equal(a, b)


def test_host_state_step_without_the_streams(gpu_lib):
    from owt import lib as owt_lib
    from owt.solver import GpuSolver
    got = []
    for limit in (-1, 0):
        s = _solver(_params(8))
        s.limit_stream_bytes(limit)
        s.set_host_chunks(3)
        hist = [s.get(n) for n in GpuSolver.HISTORY]
        means = np.array([s.get_cvec(n) for n in owt_lib.MEANS])
        got.append(s.time_Integration_host(hist, means, s.friction()))
        s.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_batch_with_a_channel_without_streams(gpu_lib):
    from owt.batch import Batch
    shapes = [dict(), dict(NX=12, NY=40), dict(NZ=10, NY=18)]
    got = []
    for limit in (None, 0):
        solvers = [_solver(_params(8, **k), seed=5 + i) for i, k in enumerate(shapes)]
        if limit is not None:
            solvers[1].limit_stream_bytes(limit)
        b = Batch(solvers)
        assert ("stream" in b.tuning_report()) == (limit is None)
        b.step(3)
        b.synchronize()
        if limit is None:  # the batch holds the addresses: they stay
            held = solvers[0].info("device_bytes")
            solvers[0].limit_stream_bytes(0)
            if "stream" in b.tuning_report().split("->")[1]:
                assert solvers[0].info("device_bytes") == held
            b.step(1)
            solvers[0].limit_stream_bytes(-1)
        else:
            b.step(1)
        b.synchronize()
        got.append([[s.get(n) for n in FIELDS] for s in solvers])
        b.close()
        for s in solvers:
            s.close()
    for x, y in zip(*got):
        for a, c in zip(x, y):
            np.testing.assert_array_equal(a, c)


def _fill(s):
    """An allocation of handle s that no device has room for."""
    from owt.lib import OwtError
    s.drag_forward(1, 10 ** 9)
    with pytest.raises(OwtError) as e:
        s.drag_backward()
    assert e.value.code == 5


def test_other_handles_give_their_streams(reference):
    """Where an allocation of one handle fails, idle handles give back their
    streams, go on with the same bits and build them again; a batch keeps its own."""
    from owt.batch import Batch
    order, ref, size = reference
    s, asking, member = _solver(_params(order)), _solver(_params(8)), _solver(_params(8), seed=4)
    s.time_Integration(2)
    asking.time_Integration(1)
    b = Batch([member])
    held = [x.info("device_bytes") for x in (s, member)]
    _fill(asking)  # the first time its own go, the second time the others'
    assert s.info("device_bytes") == held[0]
    _fill(asking)
    asking.limit_stream_bytes(0)
    _fill(asking)
    assert s.info("device_bytes") == held[0] - size
    if "stream" in b.tuning_report().split("->")[1]:
        assert member.info("device_bytes") == held[1]
    s.time_Integration(1)
    assert s.info("device_bytes") == held[0]
    _same(s, ref)
    alone = _solver(_params(8), seed=4)
    alone.time_Integration(2)
    b.step(2)
    b.synchronize()
    _same(member, alone)
    b.close()
    for x in (s, asking, member, alone):
        x.close()


def test_giving_streams_while_another_thread_steps(gpu_lib):
    import threading
    p = _params(8)
    ref, s, asking = _solver(p), _solver(p), _solver(p, seed=9)
    ref.time_Integration(200)
    asking.limit_stream_bytes(0)
    t = threading.Thread(target=lambda: [s.time_Integration(1) for _ in range(200)])
    t.start()
    while t.is_alive():
        _fill(asking)
    t.join()
    _same(s, ref)
    for x in (ref, s, asking):
        x.close()
