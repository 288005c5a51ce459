"""The calls whose speed matters, with inputs a program has in hand before them.

Each case names one public call of the library (or the short sequence a driver
loop makes) at one size: whole time steps in both precisions from a minimal
channel to the Re_tau 550 box, the 64-channel ensemble, the wall-drag gradient,
the step on a state the caller holds, and single routines.  ``listed()`` gives
the cases that are timed, ``draw(rng)`` further ones of the same ranges,
``prepare``/``run`` a case's state and one pass through it, ``work`` the bytes
and operations a pass cannot do without, and ``exact`` its results in plain
float64 where that is quick to compute.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "open-3d-wallturbulence_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from owt import lib as owt_lib  # noqa: E402
from owt.adjoint import wall_drag  # noqa: E402
from owt.batch import Batch, minimal_channels  # noqa: E402
from owt.params import CaseParams  # noqa: E402
from owt.solver import GpuSolver  # noqa: E402

# name prefix -> box: domain (through the fundamental wavenumbers), grid
# stretching, viscosity, time step.  "r180" and "r550" are the two channels of
# the tests and the benchmark (the time step of r550 is the one its 500-step
# profile test is stable with), "minimal" a minimal flow unit.
BOXES = {
    "minimal": dict(dt=0.004, dkx=1.4, dkz=4.2, alpha_mesh=2.0, nu=1.0 / 2800.0),
    "r180": dict(dt=0.005, dkx=0.5, dkz=1.5, alpha_mesh=2.0, nu=1.0 / 2800.0),
    "r550": dict(dt=0.001, dkx=1.0, dkz=2.0, alpha_mesh=2.2, nu=1.0e-4),
}


def listed():
    return [
        # The benchmark's workload: advance the Re_tau 550 box in FP64, then read the
        # velocity back as a driver does for a snapshot.
        dict(name="steps_fp64_384x257x384", kind="steps", box="r550", nx=384, ny=257, nz=384, prec="fp64", order=8,
             steps=5),
        # The same in mixed precision.
        dict(name="steps_mixed_384x257x384", kind="steps", box="r550", nx=384, ny=257, nz=384, prec="mixed", order=8,
             steps=10),
        # The Re_tau 180 channel, the size of the parity tests, in both precisions.
        dict(name="steps_fp64_128x129x128", kind="steps", box="r180", nx=128, ny=129, nz=128, prec="fp64", order=8,
             steps=20),
        dict(name="steps_mixed_128x129x128", kind="steps", box="r180", nx=128, ny=129, nz=128, prec="mixed", order=8,
             steps=20),
        # Ragged sizes (transform lines of 240 and 180 points, even NY) with the
        # sixth-order option.
        dict(name="steps_order6_160x100x120", kind="steps", box="r180", nx=160, ny=100, nz=120, prec="fp64", order=6,
             steps=10),
        # One step of a minimal flow unit and its velocity: launches and latency.
        dict(name="step_fp64_32x65x32", kind="steps", box="minimal", nx=32, ny=65, nz=32, prec="fp64", order=8,
             steps=1),
        # The 64-channel ensemble of uneven minimal channels, one graph launch a step.
        dict(name="batch64_mixed", kind="batch", channels=64, prec="mixed", steps=20, draw_seed=0),
        # Gradient of the wall drag with respect to wall blowing and suction.
        dict(name="drag_gradient_128x129x128", kind="drag", box="r180", nx=128, ny=129, nz=128, steps=20, interval=10),
        # One step on a state the caller holds in (pinned) host memory, as the
        # reference's globals are.
        dict(name="host_step_128x129x128", kind="host_step", box="r180", nx=128, ny=129, nz=128, prec="fp64"),
        # The dealiased Lamb vector alone, at the size of the reference's Re_tau 180
        # case file (lines of 480 points), and its three fields.
        dict(name="lamb_fp64_320x160x320", kind="lamb", box="r180", nx=320, ny=160, nz=320),
        # Wall-normal profiles of the current velocity, a run's usual output.
        dict(name="statistics_192x129x192", kind="statistics", box="r180", nx=192, ny=129, nz=192),
        # The wall-normal derivative on a caller's own device arrays.
        dict(name="dy1_129x4096", kind="dy1", ny=129, lines=4096, alpha_mesh=2.0),
    ]


SIZES = [16, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192,
         200, 216, 240, 250, 256, 270, 288, 300, 320, 324, 360, 384]


def _size(rng, lo, hi):
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((s for s in SIZES if s % 2 == 0), key=lambda s: abs(math.log(s / t)))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "drag", "host_step", "lamb", "statistics", "dy1"])
    if kind == "dy1":
        ny = int(round(math.exp(rng.uniform(math.log(33), math.log(513)))))
        return dict(kind=kind, ny=ny, lines=int(round(math.exp(rng.uniform(math.log(64), math.log((1 << 20) // ny - 1))))),
                    alpha_mesh=2.0)
    if kind == "batch":
        return dict(kind=kind, channels=rng.randint(8, 63), prec=rng.choice(["mixed", "mixed", "fp64"]), steps=20,
                    draw_seed=rng.randint(1, 1 << 20))
    hi = {"steps": 384, "drag": 128, "host_step": 160, "lamb": 320, "statistics": 256}[kind]
    nx, nz = _size(rng, 32, hi), _size(rng, 32, hi)
    ny = int(round(math.exp(rng.uniform(math.log(49), math.log(257 if hi >= 256 else 129)))))
    c = dict(kind=kind, box="minimal" if max(nx, nz) <= 64 else "r180" if max(nx, nz) <= 200 else "r550", nx=nx, ny=ny,
             nz=nz)
    if kind == "steps":
        points = nx * ny * nz
        c.update(prec=rng.choice(["fp64", "mixed"]), order=rng.choice([8, 8, 8, 6]),
                 steps=1 if points < 3e5 else 5 if points > 1e7 else 20)
    elif kind == "host_step":
        c.update(prec=rng.choice(["fp64", "mixed"]))
    elif kind == "drag":
        c.update(steps=rng.choice([10, 20]), interval=10)
    return c


# -- inputs -------------------------------------------------------------------


def _params(case):
    return CaseParams(NX=case["nx"], NY=case["ny"], NZ=case["nz"], fd_order=case.get("order", 8),
                      **BOXES[case["box"]]).validate()


def _pinned(shape, dtype=torch.complex128):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _velocity(p, seed):
    """Laminar flow plus a divergence-free random perturbation of RMS about 0.1
    with a k^-2 spectrum, [z][x][y] host arrays: v = (1 - y^2)^2 a, omega_y =
    (1 - y^2) b, u and w from continuity."""
    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(seed)
    NZ, NXH, NY = p.spectral_shape
    s = torch.linspace(-1.0, 1.0, NY, dtype=torch.float64, device=dev)
    y = torch.tanh(p.alpha_mesh * s) / math.tanh(p.alpha_mesh)
    kx = torch.arange(NXH, dtype=torch.float64, device=dev)[None, :] * p.dkx
    kz = torch.arange(NZ, dtype=torch.float64, device=dev)
    kz = torch.where(kz >= NZ // 2, kz - NZ, kz)[:, None] * p.dkz
    k2 = kx ** 2 + kz ** 2
    k2[0, 0] = 1.0
    amp = min(p.dkx, p.dkz) ** 2 / k2
    amp[0, 0] = 0.0
    amp[NZ // 2] = 0.0

    def random_modes():
        r = torch.randn((NZ, NXH, 2), dtype=torch.float64, device=dev, generator=gen)
        a = torch.view_as_complex(r) * amp
        a[NZ // 2 + 1:, 0] = a[1:NZ // 2, 0].flip(0).conj()  # a real field
        return a

    a0, a1, b0 = random_modes(), random_modes(), random_modes()
    q = 1.0 - y ** 2
    v = a0[..., None] * q ** 2 + a1[..., None] * (q ** 2 * y)
    dv = a0[..., None] * (-4.0 * y * q) + a1[..., None] * (q ** 2 - 4.0 * y ** 2 * q)
    g = b0[..., None] * q
    ikx, ikz = (1j * kx / k2)[..., None], (1j * kz / k2)[..., None]
    u, w = ikx * dv - ikz * g, ikx * g + ikz * dv
    rms = math.sqrt(sum(float((f.abs() ** 2).sum()) for f in (u, v, w)) * 2.0 / (3.0 * NY))
    fields = [f * (0.1 / rms) for f in (u, v, w)]
    fields[0][0, 0] = 1.5 * q
    return [f.cpu().numpy() for f in fields]


def _solver(case, seed):
    p = _params(case)
    s = GpuSolver(p, precision=case.get("prec", "fp64"))
    s.use_graph(True)
    s.init_fields(*_velocity(p, seed))
    return s, p


def _wall(p, seed):
    """Wall blowing and suction of RMS 1e-3 on both walls, [2][NZ][NXH]."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((2, p.NZ, p.NXH)) + 1j * rng.standard_normal((2, p.NZ, p.NXH))
    a[:, p.NZH] = 0.0
    a[:, 0, 0] = 0.0
    a[:, p.NZH + 1:, 0] = a[:, 1:p.NZH, 0][:, ::-1].conj()
    return a * (1e-3 / math.sqrt(2.0 * np.sum(np.abs(a) ** 2) / 2.0))


def _lamb_fields(p, seed):
    """Velocity and vorticity for the Lamb vector: the velocity above and a
    vorticity of the same spectrum, growing towards the walls."""
    vel = _velocity(p, seed)
    vor = _velocity(p, seed + 7919)
    return vel + [20.0 * f for f in vor]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dy1":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        a = torch.randn((case["ny"], case["lines"], 2), dtype=torch.float64, device="cuda", generator=gen)
        return dict(case=case, inp=a, out=torch.empty_like(a), lib=owt_lib.load())
    if kind == "batch":
        solvers = []
        for i, p in enumerate(minimal_channels(case["channels"], seed=case["draw_seed"])):
            s = GpuSolver(p, precision=case["prec"])
            s.init_fields(*_velocity(p, seed * 64 + i))
            solvers.append(s)
        return dict(case=case, solvers=solvers, batch=Batch(solvers), out=[_pinned(s.shape) for s in solvers])
    if kind == "lamb":
        p = _params(case)
        s = GpuSolver(p)
        for n, f in zip(("velx", "vely", "velz", "vorx", "vory", "vorz"), _lamb_fields(p, seed)):
            s.set(n, f)
        return dict(case=case, solver=s, out=[_pinned(s.shape) for _ in range(3)])
    s, p = _solver(case, seed)
    if kind == "statistics":
        return dict(case=case, solver=s)
    if kind == "drag":
        return dict(case=case, solver=s, start=s.checkpoint(), wall=[torch.from_numpy(a.copy()) for a in _wall(p, seed)])
    if kind == "host_step":
        hist = [s.get(n, out=_pinned(s.shape)) for n in GpuSolver.HISTORY]
        means = np.array([s.get_cvec(n) for n in owt_lib.MEANS])
        return dict(case=case, solver=s, hist=hist, means=means, fric=s.friction(),
                    out=[_pinned(s.shape) for _ in range(2)])
    s.time_Integration(1)  # a program's first step tunes and captures
    s.synchronize()
    return dict(case=case, solver=s, out=[_pinned(s.shape) for _ in range(3)])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        s = state["solver"]
        s.time_Integration(case["steps"])
        return [s.get(n, out=o) for n, o in zip(("velx", "vely", "velz"), state["out"])]
    if kind == "batch":
        state["batch"].step(case["steps"])
        state["batch"].synchronize()
        return [s.get("vely", out=o) for s, o in zip(state["solvers"], state["out"])]
    if kind == "drag":
        wb, wt = (a.clone().requires_grad_(True) for a in state["wall"])
        J = wall_drag(state["solver"], wb, wt, case["steps"], case["interval"], start=state["start"])
        J.backward()
        return dict(drag=J.detach(), bottom=wb.grad, top=wt.grad)
    if kind == "host_step":
        v, g, fric = state["solver"].time_Integration_host(state["hist"], state["means"], state["fric"], *state["out"])
        return dict(vely=v, vory=g, friction=fric)
    if kind == "lamb":
        s = state["solver"]
        s.Lamb_vec()
        return [s.get(n, out=o) for n, o in zip(("lmbx", "lmby", "lmbz"), state["out"])]
    if kind == "statistics":
        return state["solver"].statistics()
    inp, out = state["inp"], state["out"]
    rc = state["lib"].owt_dy1_noalloc(case["ny"], case["lines"], float(case["alpha_mesh"]), inp.data_ptr(),
                                      out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != owt_lib.OK:
        raise RuntimeError(state["lib"].owt_last_error(None).decode())
    return out


# -- work ---------------------------------------------------------------------


def _fft_flops(nx2, nz2, nxh, ny):
    return ny * (9 * nxh * 5 * nz2 * math.log2(nz2) + 4.5 * nz2 * 5 * nx2 * math.log2(nx2) + 9 * nz2 * nx2)


def _step_work(nx, ny, nz):
    """One step: per mode the two banded solves and the assembly around them,
    the nine dealiased transforms; the state read and written once (12 history
    fields in, 4 new levels and 4 derived fields out) and the factors once."""
    nxh, m, u = nx // 2, nx // 2 * nz, nx // 2 * (nz // 2 + 1)
    flops = m * (4 * (4 * ny + 4) * 43 + 4 * 2 * ny * 18 + 160 * ny) + _fft_flops(nx // 2 * 3, nz // 2 * 3, nxh, ny)
    return 20 * 16 * m * ny + 8 * u * ny * (4 * 25 + 2 * 12), flops


def work(case):
    kind = case["kind"]
    if kind == "dy1":
        n = case["ny"] * case["lines"]
        return {"bytes": 32 * n, "flops": 2 * 17 * n}
    if kind == "batch":
        w = [_step_work(p.NX, p.NY, p.NZ) for p in minimal_channels(case["channels"], seed=case["draw_seed"])]
        return {"bytes": case["steps"] * sum(b for b, _ in w), "flops": case["steps"] * sum(f for _, f in w)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    field = 16 * (nx // 2) * ny * nz
    if kind == "statistics":
        return {"bytes": 3 * field, "flops": 8 * 3 * field / 16}
    if kind == "lamb":
        return {"bytes": 9 * field, "flops": _fft_flops(nx // 2 * 3, nz // 2 * 3, nx // 2, ny)}
    b, f = _step_work(nx, ny, nz)
    if kind == "drag":  # forward and adjoint steps
        return {"bytes": 2 * case["steps"] * b, "flops": 2 * case["steps"] * f}
    n = case.get("steps", 1)
    return {"bytes": n * b, "flops": n * f}


# -- results in plain float64 -------------------------------------------------


def _stencils(n):
    """Compact-difference matrices A_q, B_q (q = 1..4) on n uniform nodes over
    [-1, 1]: the method's interior schemes (eighth order for the first three
    derivatives, sixth for the fourth) and boundary closures, the third
    derivative's top row with the coefficients the method runs with."""
    h = 2.0 / (n - 1.0)
    A, B = np.zeros((4, n, n)), np.zeros((4, n, n))

    def row(q, i, a, b, power, at=None, first=None):
        """a, b: {offset: value} around node `at` (default i)."""
        c = i if at is None else at
        for o, x in a.items():
            A[q, i, c + o] += x
        for o, x in b.items():
            B[q, i, c + o] += x / h ** power

    def sym(*v):
        d = {0: v[0]}
        for k, x in enumerate(v[1:], 1):
            d[k] = d[-k] = x
        return d

    def anti(*v):
        d = {}
        for k, x in enumerate(v, 1):
            d[k], d[-k] = x, -x
        return d

    for i in range(2, n - 2):
        row(0, i, sym(1, 4 / 9, 1 / 36), anti(20 / 27, 25 / 216), 1)
        row(1, i, sym(1, 344 / 1179, 23 / 2358), sym(-2 * 320 / 393 - 155 / 393, 320 / 393, 155 / 786), 2)
    for i in range(3, n - 3):
        a, b = 160 / 83, -5 / 166
        row(2, i, sym(1, 147 / 332, 1 / 166), anti(-a - 3 * b / 8, a / 2, b / 8), 3)
        a, b = 19 / 13, 1 / 13
        row(3, i, sym(1, 7 / 26), sym(6 * a + 16 * b / 6, -4 * a - 9 * b / 6, a, b / 6), 4)
    for i in (1, n - 2):
        row(0, i, sym(1, 1 / 4), anti(3 / 4), 1)
        row(1, i, sym(1, 2 / 11), sym(-24 / 11 - 3 / 22, 12 / 11, 3 / 44), 2, at=2 if i == 1 else n - 3)
    for i in (2, n - 3):
        row(2, i, sym(1, 4 / 9, 1 / 126), anti(-40 / 21, 20 / 21), 3)
        row(3, i, sym(1, 1 / 4), sym(9, -6, 3 / 2), 4)
    row(2, 1, sym(1, 1 / 2), anti(-2, 1), 3, at=2)
    row(2, n - 2, sym(1, 1 / 2), anti(-2, 1), 3, at=n - 3)
    for i, s in ((0, 1), (n - 1, -1)):  # walls, and the nodes beside them for the fourth derivative
        row(0, i, {0: 1, s: 3}, {0: -s * 17 / 6, s: s * 3 / 2, 2 * s: s * 3 / 2, 3 * s: -s / 6}, 1)
        row(1, i, {0: 1, s: 10, 2 * s: 1}, {0: 12, s: -24, 2 * s: 12}, 2)
        top = {0: -8, s: 26, 2 * s: -30, 3 * s: -2}
        row(2, i, {0: 1, s: -7}, {0: 8, 1: -26, 2: 30, 3: -14, 4: 2} if s == 1 else top, 3)
        row(3, i, {0: 1, s: -2}, {0: -1, s: 4, 2 * s: -6, 3 * s: 4, 4 * s: -1}, 4)
        row(3, i + s, {-s: 1, 0: -2, s: 7}, {-s: 6, 0: -24, s: 36, 2 * s: -24, 3 * s: 6}, 4)
    return A, B


def _derivatives(n, alpha):
    """DY1, DY2, DY4 on y = tanh(alpha s)/tanh(alpha), by the chain rule."""
    A, B = _stencils(n)
    D = [np.linalg.solve(a, b) for a, b in zip(A, B)]
    s = 2.0 * np.arange(n) / (n - 1.0) - 1.0
    t, c = np.tanh(alpha * s), 1.0 / math.tanh(alpha)
    e = 1.0 - t ** 2
    d1, d2 = alpha * c * e, -2 * alpha ** 2 * c * e * t
    d3, d4 = 2 * alpha ** 3 * c * e * (3 * t ** 2 - 1), 8 * alpha ** 4 * c * e * t * (2 - 3 * t ** 2)

    def mix(*coef):
        return sum(x[:, None] * m for x, m in zip(coef, D))

    return (mix(1 / d1), mix(-d2 / d1 ** 3, d1 ** -2.0),
            mix(-d4 / d1 ** 5 + 10 * d3 * d2 / d1 ** 6 - 15 * d2 ** 3 / d1 ** 7,
                -4 * d3 / d1 ** 5 + 15 * d2 ** 2 / d1 ** 6, -6 * d2 / d1 ** 5, d1 ** -4.0), c * t)


def _lamb(f, nx, nz):
    """Dealiased u x omega of six spectral fields [z][x][y]."""
    nxh, nzh, nx2, nz2 = nx // 2, nz // 2, nx // 2 * 3, nz // 2 * 3

    def phys(a):
        p = torch.zeros((nz2, nxh) + a.shape[2:], dtype=a.dtype, device=a.device)
        p[:nzh] = a[:nzh]
        p[nz + 1:] = a[nzh + 1:]
        p = torch.fft.ifft(p, dim=0, norm="forward")
        x = torch.zeros((nz2, nx2 // 2 + 1) + a.shape[2:], dtype=a.dtype, device=a.device)
        x[:, :nxh] = p
        return torch.fft.irfft(x, n=nx2, dim=1, norm="forward")

    def spec(p):
        z = torch.fft.fft(torch.fft.rfft(p, dim=1, norm="forward")[:, :nxh], dim=0, norm="forward")
        return torch.cat([z[:nzh], z[nz:]], dim=0)

    u, v, w, ox, oy, oz = (phys(a) for a in f)
    return [spec(v * oz - w * oy), spec(w * ox - u * oz), spec(u * oy - v * ox)]


class _Channel:
    """The method's time step with dense wall-normal matrices."""

    def __init__(self, p, vel, wall=None):
        self.p, N, dev = p, p.NY, "cuda"
        d = [torch.from_numpy(np.ascontiguousarray(m)).to(dev) for m in _derivatives(N, p.alpha_mesh)]
        D1, D2, D4 = d[:3]
        self.D1, self.D2 = D1.T.to(torch.complex128), D2.T.to(torch.complex128)
        kx = torch.arange(p.NXH, dtype=torch.float64, device=dev) * p.dkx
        kz = torch.arange(p.NZ, dtype=torch.float64, device=dev)
        kz = torch.where(kz >= p.NZH, kz - p.NZ, kz) * p.dkz
        self.kx, self.kz = kx[None, :, None], kz[:, None, None]
        self.k2 = self.kx ** 2 + self.kz ** 2
        eye = torch.eye(N, dtype=torch.float64, device=dev)
        k2, nu, g0 = self.k2[..., None], p.nu, 11.0 / (6.0 * p.dt)
        Av = -nu * D4 + (g0 + 2 * nu * k2) * D2 - (nu * k2 ** 2 + g0 * k2) * eye
        Ag = -nu * D2 + (nu * k2 + g0) * eye
        for i in (0, N - 1):
            Av[..., i, :], Ag[..., i, :] = eye[i], eye[i]
        Av[..., 1, :], Av[..., N - 2, :] = D1[0], D1[N - 1]
        self.lu = [torch.linalg.lu_factor(m) for m in (Av, Ag)]
        self.wall = None if wall is None else torch.from_numpy(wall).to(dev)
        u, v, w = (torch.from_numpy(a).to(dev) for a in vel)
        ox, oy, oz = w @ self.D1 - 1j * self.kz * v, 1j * self.kz * u - 1j * self.kx * w, 1j * self.kx * v - u @ self.D1
        self.f = [u, v, w, ox, oy, oz]
        self.v, self.g = [v] * 3, [oy] * 3
        self.mean = [[u[0, 0]] * 3, [w[0, 0]] * 3]
        self.fric = [[self._force(m[0])] * 3 for m in self.mean]
        self.hv, self.hg, self.lm = [None] * 3, [None] * 3, [[None] * 3, [None] * 3]
        self._nonlinear(start=True)

    def _force(self, m):
        d = m @ self.D1
        return -0.5 * self.p.nu * (d[-1] - d[0]).real

    def _nonlinear(self, start=False):
        lx, ly, lz = _lamb(self.f, self.p.NX, self.p.NZ)
        hv = -self.k2 * ly - (1j * self.kx * lx + 1j * self.kz * lz) @ self.D1
        hg = 1j * self.kz * lx - 1j * self.kx * lz
        if start:
            self.hv, self.hg, self.lm = [hv] * 3, [hg] * 3, [[lx[0, 0]] * 3, [lz[0, 0]] * 3]
        else:
            self.hv, self.hg = [hv] + self.hv[:2], [hg] + self.hg[:2]
            self.lm = [[a[0, 0]] + old[:2] for a, old in zip((lx, lz), self.lm)]

    def step(self):
        p, dt = self.p, self.p.dt

        def al(h):
            return (3.0 * h[0] - 1.5 * h[1] + h[2] / 3.0) / dt

        def be(h):
            return 3.0 * h[0] - 3.0 * h[1] + h[2]

        vs = al(self.v)
        rv = be(self.hv) - self.k2 * vs + vs @ self.D2
        rg = be(self.hg) + al(self.g)
        rv[..., :2], rv[..., -2:], rg[..., :1], rg[..., -1:] = 0, 0, 0, 0
        if self.wall is not None:
            rv[..., 0], rv[..., -1] = self.wall[0], self.wall[1]

        def solve(lu, r):
            x = torch.linalg.lu_solve(*lu, torch.stack([r.real, r.imag], dim=-1).contiguous())
            return torch.complex(x[..., 0], x[..., 1])

        v, g = solve(self.lu[0], rv), solve(self.lu[1], rg)
        d1, d2, dg = v @ self.D1, v @ self.D2, g @ self.D1
        safe = torch.where(self.k2 < 1e-8, 1.0, self.k2)
        ix, iz = 1j * self.kx / safe, 1j * self.kz / safe
        u, w = ix * d1 - iz * g, ix * g + iz * d1
        ox, oz = ix * dg + iz * (d2 - self.k2 * v), iz * dg - ix * (d2 - self.k2 * v)
        new = []
        for m, l, f in zip(self.mean, self.lm, self.fric):
            r = be([a + b for a, b in zip(l, f)]) + al(m)
            r[0] = r[-1] = 0
            new.append(solve([a[0, 0] for a in self.lu[1]], r))
        u[0, 0], w[0, 0], ox[0, 0], oz[0, 0] = new[0], new[1], new[1] @ self.D1, -(new[0] @ self.D1)
        self.f = [u, v, w, ox, g, oz]
        self.v, self.g = [v] + self.v[:2], [g] + self.g[:2]
        self.mean = [[a] + old[:2] for a, old in zip(new, self.mean)]
        self.fric = [[self._force(a)] + old[:2] for a, old in zip(new, self.fric)]
        self._nonlinear()


def _host(fields):
    return [f.cpu().numpy() for f in fields]


def exact(case, seed):
    kind = case["kind"]
    if kind == "dy1":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        a = torch.randn((case["ny"], case["lines"], 2), dtype=torch.float64, device="cuda", generator=gen)
        d1 = torch.from_numpy(_derivatives(case["ny"], case["alpha_mesh"])[0]).to(a)
        return (d1 @ a.reshape(case["ny"], -1)).reshape(a.shape)
    if kind == "batch":  # the first channels; the others take long
        out = [None] * case["channels"]
        for i, p in list(enumerate(minimal_channels(case["channels"], seed=case["draw_seed"])))[:4]:
            c = _Channel(p, _velocity(p, seed * 64 + i))
            for _ in range(case["steps"]):
                c.step()
            out[i] = c.f[1].cpu().numpy()
        return out
    p = _params(case)
    if kind == "lamb":
        return _host(_lamb([torch.from_numpy(f).cuda() for f in _lamb_fields(p, seed)], p.NX, p.NZ))
    if kind == "statistics":
        u, v, w = (torch.from_numpy(a).cuda() for a in _velocity(p, seed))

        def mean(a, b):  # over x and z; kx > 0 stands for the conjugate half too, the Nyquist kz row for nothing
            t = (a * b.conj()).real
            t[p.NZH] = 0
            return (2.0 * t[:, 1:].sum(dim=(0, 1)) + t[:, 0].sum(dim=0))

        U, V, W = (a[0, 0].real for a in (u, v, w))
        rms = [torch.sqrt(torch.clamp(mean(a, a) - m ** 2, min=0.0)) for a, m in ((u, U), (v, V), (w, W))]
        return dict(zip(GpuSolver.STAT_NAMES, _host([U, V, W] + rms + [mean(u, v) - U * V])))
    # dense matrices of every mode: both systems held twice over have to fit
    if case.get("order", 8) != 8 or p.NZ * p.NXH * p.NY ** 2 > 3e8:
        return None
    c = _Channel(p, _velocity(p, seed), _wall(p, seed) if kind == "drag" else None)
    if kind == "drag":
        J = 0.0
        for _ in range(case["steps"]):
            c.step()
            J += float(c.fric[0][0]) / case["steps"]
        return dict(drag=J, bottom=None, top=None)
    if kind == "host_step":
        c.step()
        return dict(vely=c.f[1].cpu().numpy(), vory=c.f[4].cpu().numpy(),
                    friction=np.array([float(x) for f in c.fric for x in f]))
    for _ in range(case["steps"] + 1):
        c.step()
    return _host(c.f[:3])
