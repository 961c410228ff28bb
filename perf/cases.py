"""What a user of lex_gb300 has it do, as cases that can be timed and compared.

Kinds of case, each through the package's public entry points:

  step       a sprint: state in, `steps` RK3 big steps (one captured graph each), state out, all as
             CUDA tensors in the device layout (lex_gb300.autograd.set_state / get_state, Solver.step)
  host       one big step between pinned host buffers in the reference's padded layout, as a driver
             that owns the state on the host calls it (Solver.upload_ptrs / step / download_ptrs)
  grad       a differentiable rollout and its reverse pass: the adjoint of the initial state and of
             the Smagorinsky constant (lex_gb300.autograd.rollout)
  corrected  a sprint with the learned SGS correction inside the step graph (lex_gb300.sgs_cnn.attach)
  net        forward and backward of the correction's network, as training runs it
             (lex_gb300.sgs_cnn.net_apply)

States are a warm bubble (1 to 3 K) on the neutral 300 K base state with exponential humidity, with
winds, pi' and humidity perturbations of a developed run: a few horizontal waves plus grid noise.
`exact` restates the model in FP64 with plain torch on the interior grid.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from lex_gb300 import autograd as lag
from lex_gb300 import sgs_cnn
from lex_gb300.solver import Solver

# spacings and big steps of the package's own configurations: (dx = dy, dz, dt)
SPACINGS = {"100m": (100.0, 100.0, 1.0), "300m": (300.0, 150.0, 2.0), "600m": (600.0, 300.0, 3.0)}
N_SOUND = 32
CS = float(np.float32(0.18))
THETA_REF = 300.0


def listed():
    return [
        # the smallest call: one step of the smoke-test grid, all launch latency
        dict(name="step_16x16x12", kind="step", nx=16, ny=16, nz=12, spacing="600m", turb=1, cor=0, steps=1),
        # the coarse run between two saves (10 steps of 3 s), launch- and latency-bound
        dict(name="sprint_32x32x32", kind="step", nx=32, ny=32, nz=32, spacing="600m", turb=1, cor=0, steps=10),
        # the mid-size grid of the gradient check
        dict(name="steps_64x64x64", kind="step", nx=64, ny=64, nz=64, spacing="300m", turb=1, cor=0, steps=5),
        # a grid nobody rounded: nx not a multiple of 4, odd ny and nz, with Coriolis
        dict(name="steps_101x75x59", kind="step", nx=101, ny=75, nz=59, spacing="300m", turb=1, cor=1, steps=2),
        # the benchmark's high-resolution warm bubble
        dict(name="steps_192x192x96", kind="step", nx=192, ny=192, nz=96, spacing="100m", turb=1, cor=0, steps=2),
        # the namelist's default grid, without SGS, with Coriolis and the large-scale pressure gradient
        dict(name="step_240x240x120", kind="step", nx=240, ny=240, nz=120, spacing="100m", turb=0, cor=2, steps=1),
        # the benchmark's grid with the state on the host every step (coupled or saved each step)
        dict(name="host_192x192x96", kind="host", nx=192, ny=192, nz=96, spacing="100m", turb=1, cor=0, f64=False),
        # two steps of the gradient check's rollout: the last step's intermediates are kept, the first recomputed
        dict(name="grad_64x64x64", kind="grad", nx=64, ny=64, nz=64, spacing="300m", turb=1, cor=0, steps=2),
        # forward and adjoint of one high-resolution step
        dict(name="grad_192x192x96", kind="grad", nx=192, ny=192, nz=96, spacing="100m", turb=1, cor=0, steps=1),
        # the larger learned-SGS run's corrected steps
        dict(name="corrected_128x128x64", kind="corrected", nx=128, ny=128, nz=64, spacing="600m", turb=1, cor=0,
             steps=2),
        # a training pass of the network on the coarse grid
        dict(name="net_32x32x32", kind="net", nx=32, ny=32, nz=32),
        # and on the larger learned-SGS grid
        dict(name="net_128x128x64", kind="net", nx=128, ny=128, nz=64),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "host", "grad", "grad", "corrected", "net"])
    most = {"step": 240 * 240 * 120, "host": 192 * 192 * 96, "grad": 192 * 192 * 96, "corrected": 128 * 128 * 64,
            "net": 128 * 128 * 64}[kind]
    while True:
        nx, ny, nz = _log_size(rng, 16, 240), _log_size(rng, 16, 240), _log_size(rng, 12, 120)
        if kind in ("corrected", "net"):          # the convolutions take nx in multiples of 16
            nx = max(16, nx // 16 * 16)
        elif rng.random() < 0.6:                  # most users pick a multiple of 4 or more
            nx = max(16, nx // 4 * 4)
        if nx * ny * nz <= most:
            break
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "net":
        return c
    c.update(spacing=rng.choice(sorted(SPACINGS)), turb=rng.choice([0, 1, 1]), cor=rng.choice([0, 0, 1, 2]))
    if kind == "host":
        c["f64"] = rng.random() < 0.3
    elif kind == "grad":
        c["steps"] = rng.randint(1, 2) if nx * ny * nz < 64 ** 3 else 1
    else:
        c["steps"] = max(1, min(10, most // (nx * ny * nz)))
    return c


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _columns(case):
    """Padded FP64 theta0 and qv0 columns (one ghost level at either end)."""
    nz, dz = case["nz"], SPACINGS[case["spacing"]][1]
    z = (np.arange(nz + 2) - 0.5) * dz
    return np.full(nz + 2, THETA_REF), 0.014 * np.exp(-z / 2500.0)


def _waves(gen, shape, vertical):
    """A few horizontal waves times a vertical profile, of unit size, plus grid noise of one percent."""
    n, ny, nx = shape
    g = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)
    x = 2 * math.pi * torch.arange(nx, device="cuda", dtype=torch.float64) / nx
    y = 2 * math.pi * torch.arange(ny, device="cuda", dtype=torch.float64) / ny
    z = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    out = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for m in range(1, 4):
        a = g(4).tolist()
        prof = torch.sin(math.pi * m * z) if vertical else torch.cos(math.pi * m * z + 6.28 * a[0])
        wave = torch.sin(m * x + 6.28 * a[1])[None, :] * torch.cos((4 - m) * y + 6.28 * a[2])[:, None]
        out += (0.4 + 0.6 * a[3]) * prof[:, None, None] * wave[None]
    return out + 0.01 * torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _state(case, seed):
    """The six FP32 fields in the device layout, theta relative to THETA_REF."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = _generator(seed)
    cells, faces = (nz, ny, nx), (nz + 1, ny, nx)
    f64 = dict(device="cuda", dtype=torch.float64)
    amp = 1.0 + 2.0 * float(torch.rand(1, generator=gen, device="cuda"))
    x = (torch.arange(nx, **f64) + 0.5) / nx - 0.5
    y = (torch.arange(ny, **f64) + 0.5) / ny - 0.5
    z = (torch.arange(nz, **f64) + 0.5) / nz - 0.25
    r = torch.sqrt((x / 0.2)[None, None, :] ** 2 + (y / 0.2)[None, :, None] ** 2 + (z / 0.2)[:, None, None] ** 2)
    T = torch.where(r <= 1.0, amp * torch.cos(0.5 * math.pi * r) ** 2, torch.zeros_like(r))
    T = T + 0.01 * (2.0 * torch.rand(cells, generator=gen, **f64) - 1.0)
    u, v = 4.0 * _waves(gen, cells, False), 4.0 * _waves(gen, cells, False)
    w = 1.5 * _waves(gen, faces, True)
    w[0] = 0.0
    w[-1] = 0.0
    p = 1.0e-4 * _waves(gen, cells, False)
    q0 = torch.as_tensor(_columns(case)[1][1:-1], **f64)[:, None, None]
    q = q0 * (1.0 + 0.03 * _waves(gen, cells, False) + 0.003 * torch.randn(cells, generator=gen, **f64))
    return tuple(a.float().contiguous() for a in (T, u, v, w, p, q))


def _solver(case):
    dx, dz, dt = SPACINGS[case["spacing"]]
    S = Solver(case["nx"], case["ny"], case["nz"], dx, dx, dz, dt, N_SOUND, turb_opt=case["turb"],
               cor_opt=case["cor"], cs=CS)
    S.integrate_base_state(*_columns(case))
    return S


def _seeds(case, seed):
    """Output adjoints: smooth fields over the size of each output field."""
    gen = _generator(seed + 77)
    cells, faces = (case["nz"], case["ny"], case["nx"]), (case["nz"] + 1, case["ny"], case["nx"])
    size = (1.0, 0.2, 0.2, 0.5, 1.0e3, 100.0)
    return tuple((s * _waves(gen, faces if f == 3 else cells, f == 3)).float() for f, s in enumerate(size))


def _net(seed, last):
    """The network with random weights; `last` scales its last layer (a trained correction is small)."""
    net = sgs_cnn.SGSNet(seed=int(seed) % 100003, zero_last=False)
    net.w[3] = net.w[3] * last
    gen = torch.Generator().manual_seed(int(seed) + 5)
    for li, (_, cout, _) in enumerate(sgs_cnn.LAYERS):
        net.b[li] = torch.where(torch.arange(cout) < (5 if li == 3 else cout),
                                0.1 * torch.randn(cout, generator=gen), torch.zeros(cout)).cuda()
    net.b[3] = net.b[3] * last
    net.refresh()
    return net


def _scale(x):
    """Input minimum and range per level, output range per point (1 % of the level's range), theta in K."""
    lo, rin, rout = [], [], []
    nz, ny, nx = x[0].shape
    for f, margin in ((0, 0.01), (1, 0.01), (2, 0.01), (3, 0.01), (5, 1.0e-5)):
        a = x[f] + THETA_REF if f == 0 else x[f]
        mn, mx = a.amin(dim=(1, 2)), a.amax(dim=(1, 2))
        if f != 3:
            mn, mx = torch.cat([mn, mn[-1:]]), torch.cat([mx, mx[-1:]])
        lo.append(mn)
        rin.append(mx - mn + margin)
        rout.append((0.01 * (mx - mn))[:, None, None].expand(nz + 1, ny, nx))
    return {"lo": torch.stack(lo), "rin": torch.stack(rin), "rout": torch.stack(rout).contiguous()}


def _net_inputs(case, seed):
    gen = _generator(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    x = torch.stack([(0.5 + 0.25 * _waves(gen, shape, False)).reshape(-1) for _ in range(5)], 1).float()
    gy = torch.stack([(0.1 * (0.5 + _waves(gen, shape, False))).reshape(-1) for _ in range(5)], 1).float()
    return x, gy


def _pad(a, field):
    """Interior [x][y][z] -> the padded layout: 3 periodic ghost cells in x and y, 1 edge copy in z;
    u and v with their duplicated periodic face."""
    cat = torch.cat
    if field == 1:
        a = cat((a, a[:1]), 0)
        a = cat((a[-4:-1], a, a[1:4]), 0)
    else:
        a = cat((a[-3:], a, a[:3]), 0)
    if field == 2:
        a = cat((a, a[:, :1]), 1)
        a = cat((a[:, -4:-1], a, a[:, 1:4]), 1)
    else:
        a = cat((a[:, -3:], a, a[:, :3]), 1)
    return cat((a[:, :, :1], a, a[:, :, -1:]), 2)


def _padded(x, theta):
    """Device-layout fields -> padded fields, `theta` added to the first."""
    return [_pad(a.permute(2, 1, 0) + (theta if f == 0 else 0.0), f) for f, a in enumerate(x)]


def _host_fields(case, seed):
    """The padded host state: theta in K, in the case's type."""
    dtype = torch.float64 if case["f64"] else torch.float32
    x = [a.double() for a in _state(case, seed)]
    return [a.to(dtype).contiguous().cpu() for a in _padded(x, THETA_REF)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "net":
        s["net"] = _net(seed, 1.0)
        s["x"], s["gy"] = _net_inputs(case, seed)
        s["x"].requires_grad_(True)
        for t in s["net"].params():
            t.requires_grad_(True)
        return s
    s["solver"] = _solver(case)
    if kind == "host":
        s["in"] = [a.pin_memory() for a in _host_fields(case, seed)]
        s["out"] = [torch.zeros_like(a).pin_memory() for a in s["in"]]
        return s
    s["x"] = _state(case, seed)
    if kind == "grad":
        for t in s["x"]:
            t.requires_grad_(True)
        s["cs"] = torch.tensor(CS, device="cuda", dtype=torch.float32, requires_grad=True) if case["turb"] else None
        s["gy"] = _seeds(case, seed)
    if kind == "corrected":
        s["net"] = _net(seed, 0.3)
        s["scale"] = _scale(s["x"])
        sgs_cnn.attach(s["solver"], s["net"], s["scale"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "net":
        out = sgs_cnn.net_apply(s["net"], s["x"], (case["nx"], case["ny"], case["nz"]))
        grads = torch.autograd.grad(out, [s["x"]] + s["net"].params(), grad_outputs=s["gy"])
        return [out.detach()] + list(grads)
    S = s["solver"]
    if kind == "host":
        S.upload_ptrs([a.data_ptr() for a in s["in"]], case["f64"])
        S.step(1)
        S.download_ptrs([a.data_ptr() for a in s["out"]], case["f64"])
        return s["out"]
    if kind == "grad":
        y = lag.rollout(S, s["x"], case["steps"], s["cs"], raw=True)
        wrt = list(s["x"]) + ([s["cs"]] if s["cs"] is not None else [])
        return [a.detach() for a in y] + list(torch.autograd.grad(y, wrt, grad_outputs=s["gy"]))
    lag.set_state(S, s["x"], raw=True)
    S.step(case["steps"])
    return list(lag.get_state(S, raw=True))


# floating-point operations a grid point of one big step takes: three stages of five WENO5 fields in
# three directions and their divergences, 49 acoustic sub-steps, Smagorinsky
FLOPS_STEP, FLOPS_SGS = 3 * (15 * 75 + 120) + 49 * 60, 450
FLOPS_NET = 2 * 27 * (5 * 32 + 2 * 32 * 32 + 32 * 5)


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "net":      # forward, input gradients and weight gradients
        return {"bytes": n * 4 * (5 + 5 + 5 + 5), "flops": 3 * n * FLOPS_NET}
    flops = n * (FLOPS_STEP + FLOPS_SGS * case["turb"])
    if kind == "host":     # the state in and out
        return {"bytes": 12 * n * (8 if case["f64"] else 4), "flops": flops}
    if kind == "grad":     # state in, state out, adjoint in, adjoint out; the reverse costs twice the forward
        return {"bytes": 24 * n * 4, "flops": 3 * case["steps"] * flops}
    if kind == "corrected":
        return {"bytes": (12 + 5) * n * 4, "flops": case["steps"] * (flops + n * FLOPS_NET)}
    return {"bytes": 12 * n * 4, "flops": case["steps"] * flops}


# ------------------------------------------------------------------------------------------------
# the same results in FP64 with plain torch: interior fields [z][y][x], u on west faces, v on south
# faces, w on faces 0..nz
# ------------------------------------------------------------------------------------------------
RD, RV, CP, G, P00 = 287.04, 461.5, 1004.64, 9.80616, 100000.0
CV, REPS = CP - RD, RV / RD


def _weno5(a, b, c, d, e, eps):
    b1 = 13.0 / 12.0 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b2 = 13.0 / 12.0 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b3 = 13.0 / 12.0 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tau = (b1 - b3).abs()
    w1, w2, w3 = (g * (1.0 + (tau / (bk + eps)).clamp_max(1e30) ** 2) for g, bk in ((0.1, b1), (0.6, b2), (0.3, b3)))
    s = w1 * (2 * a - 7 * b + 11 * c) + w2 * (-b + 5 * c + 2 * d) + w3 * (2 * c + 5 * d - e)
    return s / (6.0 * (w1 + w2 + w3))


def _weno3(a, b, c, eps):
    b1, b2 = (a - b) ** 2, (b - c) ** 2
    tau = (b1 - b2).abs()
    w1, w2 = (g * (1.0 + (tau / (bk + eps)).clamp_max(1e30) ** 2) for g, bk in ((1.0 / 3.0, b1), (2.0 / 3.0, b2)))
    return (w1 * (-0.5 * a + 1.5 * b) + w2 * (0.5 * b + 0.5 * c)) / (w1 + w2)


def _lateral(s, m, dim, eps):
    """m times the upwind value at the faces between entries i-1 and i along a periodic axis."""
    at = lambda o: torch.roll(s, -o, dim)
    pos = _weno5(at(-3), at(-2), at(-1), s, at(1), eps)
    neg = _weno5(at(2), at(1), s, at(-1), at(-2), eps)
    return torch.where(m >= 0, m * pos, m * neg)


def _vertical(s, m, eps):
    """m times the upwind value at the inner faces 1..n-1 of an n-entry column, zero faces around them."""
    n = s.shape[0]
    five = [s[o:n - 4 + o] for o in range(5)]
    up = torch.cat([0.5 * (s[:1] + s[1:2]), _weno3(s[0:1], s[1:2], s[2:3], eps), _weno5(*five, eps),
                    _weno3(s[n - 3:n - 2], s[n - 2:n - 1], s[n - 1:], eps)])
    dn = torch.cat([_weno3(s[2:3], s[1:2], s[0:1], eps), _weno5(*five[::-1], eps),
                    _weno3(s[n - 1:], s[n - 2:n - 1], s[n - 3:n - 2], eps), 0.5 * (s[n - 1:] + s[n - 2:n - 1])])
    f = torch.where(m >= 0, m * up, m * dn)
    z = torch.zeros_like(s[:1])
    return torch.cat([z, f, z])


def _mid(a):
    return 0.5 * (a[1:] + a[:-1])


def _ends(a):
    return (1.875 * a[:1] - 1.25 * a[1:2] + 0.375 * a[2:3], 1.875 * a[-1:] - 1.25 * a[-2:-1] + 0.375 * a[-3:-2])


def _im(a):
    return torch.roll(a, 1, 2)


def _ip(a):
    return torch.roll(a, -1, 2)


def _jm(a):
    return torch.roll(a, 1, 1)


def _jp(a):
    return torch.roll(a, -1, 1)


def _closed(a):
    """Values on the inner faces with zero faces below and above."""
    z = torch.zeros_like(a[:1])
    return torch.cat([z, a, z])


class _Model:
    def __init__(self, case, cs=CS):
        self.case, self.cs = case, cs
        self.dx, self.dz, self.dt = SPACINGS[case["spacing"]]
        theta0, qv0 = _columns(case)
        trho0 = theta0 * (1.0 + REPS * qv0) / (1.0 + qv0)
        faces = np.concatenate(([1.0], np.cumsum((-G / CP / trho0)[1:-1]) * self.dz + 1.0))
        pi0 = 0.5 * (faces[:-1] + faces[1:])
        rho = pi0 ** (CV / RD) * P00 / RD / trho0[1:-1]
        col = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")[:, None, None]
        self.rho, self.pi0, self.trho0 = col(rho), col(pi0), col(trho0[1:-1])
        self.rw = _mid(self.rho)                      # inner faces
        self.dpi0 = (self.pi0[1:] - self.pi0[:-1]) / self.dz

    def conv(self, fx, fy, fz):
        return -((_ip(fx) - fx) / self.dx + (_jp(fy) - fy) / self.dx + (fz[1:] - fz[:-1]) / self.dz)

    def slow(self, x):
        T, u, v, w, _, q = x
        r, rw, c = self.rho, self.rw, self.case
        dx, dz = self.dx, self.dz
        mw = rw * w[1:-1]
        mwc = _closed(mw)
        div = (_ip(r * u) - r * u) / dx + (_jp(r * v) - r * v) / dx + (mwc[1:] - mwc[:-1]) / dz
        out = []
        for s, eps in ((T, 1e-17), (q, 1e-18)):
            a = self.conv(_lateral(s, r * u, 2, eps), _lateral(s, r * v, 1, eps), _vertical(s, mw, eps))
            out.append((a + s * div) / r)
        e = 1e-16
        fx = _ip(_lateral(u, 0.5 * r * (_im(u) + u), 2, e))      # at cell i, between faces i and i+1
        fy = _lateral(u, 0.5 * r * (_im(v) + v), 1, e)
        fz = _vertical(u, 0.5 * (_im(mw) + mw), e)
        au = -((fx - _im(fx)) / dx + (_jp(fy) - fy) / dx + (fz[1:] - fz[:-1]) / dz)
        au = (au + u * 0.5 * (_im(div) + div)) / r
        fx = _lateral(v, 0.5 * r * (_jm(u) + u), 2, e)
        fy = _jp(_lateral(v, 0.5 * r * (_jm(v) + v), 1, e))
        fz = _vertical(v, 0.5 * (_jm(mw) + mw), e)
        av = -((_ip(fx) - fx) / dx + (fy - _jm(fy)) / dx + (fz[1:] - fz[:-1]) / dz)
        av = (av + v * 0.5 * (_jm(div) + div)) / r
        wi = w[1:-1]
        fx, fy = _lateral(wi, _mid(r * u), 2, e), _lateral(wi, _mid(r * v), 1, e)
        fz = _vertical(w, _mid(w) * r, e)[1:-1]                  # at cells 0..nz-1
        aw = -((_ip(fx) - fx) / dx + (_jp(fy) - fy) / dx + (fz[1:] - fz[:-1]) / dz)
        aw = (aw + wi * _mid(div)) / rw
        if c["cor"]:
            f = 1.0e-4
            au = au + f * 0.25 * (_im(v) + _jp(_im(v)) + v + _jp(v))
            av = av - f * (0.25 * (_jm(u) + _ip(_jm(u)) + u + _ip(u)) - (1.0 if c["cor"] == 2 else 0.0))
        theta = THETA_REF + T
        trho = theta * (1.0 + REPS * q) / (1.0 + q)
        aw = aw + _mid(G * (trho - self.trho0) / self.trho0)
        return out[0], au, av, aw, out[1], trho

    def smagorinsky(self, x):
        T, u, v, w, _, q = x
        r, rw, dx, dz = self.rho, self.rw, self.dx, self.dz
        theta = THETA_REF + T
        corner = lambda e: 0.25 * (e + _ip(e) + _jp(e) + _ip(_jp(e)))
        s11, s22, s33 = (_ip(u) - u) / dx, (_jp(v) - v) / dx, (w[1:] - w[:-1]) / dz
        s12 = corner(0.5 * ((u - _jm(u)) / dx + (v - _im(v)) / dx))

        def shear(h, along):
            e = 0.5 * ((h[1:] - h[:-1]) / dz + (w[1:-1] - along[0](w[1:-1])) / dx)
            b, t = _ends(e)
            e = torch.cat([b, _mid(e), t])
            return 0.5 * (e + along[1](e))
        s13, s23 = shear(u, (_im, _ip)), shear(v, (_jm, _jp))
        s2 = 2 * (s11 ** 2 + s22 ** 2 + s33 ** 2) + 4 * (s12 ** 2 + s13 ** 2 + s23 ** 2)
        tv = theta * (1.0 + (REPS - 1.0) * q)
        nf = torch.log(tv[1:] / tv[:-1]) / dz * G
        b, t = _ends(nf)
        m = s2 - 3.0 * torch.cat([b, _mid(nf), t])
        on = m > 0
        km = self.cs ** 2 * (dx * dx * dz) ** (2.0 / 3.0) * torch.where(on, torch.sqrt(torch.where(on, m, 1.0)), 0.0)
        kh = 3.0 * km
        t11, t22, t33, t12, t13, t23 = (-2.0 * km * r * s for s in (s11, s22, s33, s12, s13, s23))
        d = (t12 - _jm(t12)) / dx
        e13, e23 = _closed(_mid(t13)), _closed(_mid(t23))
        d13, d23 = (e13[1:] - e13[:-1]) / dz, (e23[1:] - e23[:-1]) / dz
        gu = -((t11 - _im(t11)) / dx + 0.25 * (_im(d) + d + _jp(_im(d)) + _jp(d)) + 0.5 * (_im(d13) + d13)) / r
        d = (t12 - _im(t12)) / dx
        gv = -(0.25 * (_jm(d) + d + _ip(_jm(d)) + _ip(d)) + (t22 - _jm(t22)) / dx + 0.5 * (_jm(d23) + d23)) / r
        gw = -(_mid((_ip(t13) - _im(t13)) / (2 * dx)) + _mid((_jp(t23) - _jm(t23)) / (2 * dx))
               + (t33[1:] - t33[:-1]) / dz) / rw

        def scalar(s):
            fx = -r * 0.5 * (kh + _im(kh)) * (s - _im(s)) / dx
            fy = -r * 0.5 * (kh + _jm(kh)) * (s - _jm(s)) / dx
            fz = _closed(-rw * _mid(kh) * (s[1:] - s[:-1]) / dz)
            return self.conv(fx, fy, fz) / r
        return gu, gv, gw, scalar(theta), scalar(q)

    def acoustic(self, u, v, w, p, ps, ru, rv, rw_, trho, n, dtau):
        dx, dz = self.dx, self.dz
        sx, sy = (ps - _im(ps)) / dx, (ps - _jm(ps)) / dx
        sz = self.dpi0 + (ps[1:] - ps[:-1]) / dz
        tx, ty, tz = (0.5 * CP * (trho + _im(trho)) / dx, 0.5 * CP * (trho + _jm(trho)) / dx,
                      0.5 * CP * (trho[1:] + trho[:-1]) / dz)
        k = RD / CV * (self.pi0 + ps)
        for _ in range(n):
            u = u + (ru - tx * (p - _im(p))) * dtau
            v = v + (rv - ty * (p - _jm(p))) * dtau
            wi = w[1:-1] + (rw_ - tz * (p[1:] - p[:-1])) * dtau
            w = _closed(wi)
            div = (_ip(u) - u) / dx + (_jp(v) - v) / dx + (w[1:] - w[:-1]) / dz
            ax, ay, az = u * sx, v * sy, _closed(0.5 * wi * sz * self.rw)
            adv = 0.5 * (ax + _ip(ax)) + 0.5 * (ay + _jp(ay)) + (az[1:] + az[:-1]) / self.rho
            p = p - 1.1 * dtau * (k * div + adv)
        return u, v, w, p

    def stage(self, dts, n, dtau, x0, xs, sgs):
        dT, ru, rv, rw_, dq, trho = self.slow(xs)
        if sgs is not None:
            ru, rv, rw_ = ru + sgs[0], rv + sgs[1], rw_ + sgs[2]
            dT, dq = dT + sgs[3], dq + sgs[4]
        u, v, w, p = self.acoustic(x0[1], x0[2], x0[3], x0[4], xs[4], ru, rv, rw_, trho, n, dtau)
        return x0[0] + dts * dT, u, v, w, p, x0[5] + dts * dq

    def step(self, x, recompute=False):
        """One big step; recompute: keep only each stage's input for the reverse pass."""
        call = (lambda f, *a: checkpoint(f, *a, use_reentrant=False)) if recompute else (lambda f, *a: f(*a))
        sgs = call(self.smagorinsky, x) if self.case["turb"] else None
        xs = x
        for dts, n in ((self.dt / 3, 1), (self.dt / 2, N_SOUND // 2), (self.dt, N_SOUND)):
            xs = call(self.stage, dts, n, dts if n == 1 else self.dt / N_SOUND, x, xs, sgs)
        return xs


def _conv(x, w, b, shape):
    """3x3x3 zero-padded convolution of [npts][cin] with w [27][cout][cin]."""
    nz, ny, nx = shape
    a = torch.nn.functional.pad(x.reshape(nz, ny, nx, -1), (0, 0, 1, 1, 1, 1, 1, 1))
    y = b.expand(nz * ny * nx, -1)
    for o in range(27):
        z0, y0, x0 = o // 9, o // 3 % 3, o % 3
        y = y + a[z0:z0 + nz, y0:y0 + ny, x0:x0 + nx].reshape(-1, a.shape[-1]) @ w[o].t()
    return y


def _layers(net):
    """The network's BF16 weights and FP32 biases as FP64 tensors."""
    return [t.detach().double() for t in net.wbf], [t.detach().double() for t in net.b]


def _apply(x, ws, bs, shape):
    a = torch.nn.functional.pad(x, (0, 16 - x.shape[1]))
    for li in range(4):
        a = checkpoint(_conv, a, ws[li], bs[li], shape, use_reentrant=False)
        if li < 3:
            a = torch.nn.functional.gelu(a, approximate="tanh")
    return a[:, :5]


def _correct(x, ws, bs, scale):
    T, u, v, w, p, q = x
    shape = T.shape
    lo, rin, rout = (scale[k].double() for k in ("lo", "rin", "rout"))
    nz = shape[0]
    n = lambda a, f, m: (a - lo[f, :m, None, None]) / rin[f, :m, None, None]
    un, vn, wn = n(u, 1, nz), n(v, 2, nz), n(w, 3, nz + 1)
    cols = (n(T + THETA_REF, 0, nz), 0.5 * (un + _ip(un)), 0.5 * (vn + _jp(vn)), _mid(wn), n(q, 4, nz))
    c = _apply(torch.stack([a.reshape(-1) for a in cols], 1), ws, bs, shape)
    c = [c[:, i].reshape(shape) for i in range(5)]
    cu, cv = 0.5 * (c[1] + _im(c[1])), 0.5 * (c[2] + _jm(c[2]))
    cu = torch.cat([cu[:, :, -1:], cu[:, :, 1:]], 2)
    cv = torch.cat([cv[:, -1:], cv[:, 1:]], 1)
    return (T + c[0] * rout[0, :nz], u + cu * rout[1, :nz], v + cv * rout[2, :nz], w + _closed(_mid(c[3])) * rout[3],
            p, q + c[4] * rout[4, :nz])


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        net = _net(seed, 1.0)
        x, gy = _net_inputs(case, seed)
        ws, bs = _layers(net)
        x = x.double().requires_grad_(True)
        for t in ws + bs:
            t.requires_grad_(True)
        out = _apply(x, ws, bs, (case["nz"], case["ny"], case["nx"]))
        return [out.detach()] + list(torch.autograd.grad(out, [x] + ws + bs, grad_outputs=gy.double()))
    if kind == "host":
        with torch.no_grad():
            back = [a.double().cuda() for a in _host_fields(case, seed)]
            x = []
            for f, a in enumerate(back):
                nx, ny = case["nx"], case["ny"]
                a = a[3:3 + nx, 3:3 + ny, 1:-1].permute(2, 1, 0).contiguous()
                x.append(a - THETA_REF if f == 0 else a)
            return [a.cpu() for a in _padded(_Model(case).step(tuple(x)), THETA_REF)]
    x = tuple(a.double() for a in _state(case, seed))
    if kind == "grad":
        for t in x:
            t.requires_grad_(True)
        cs = torch.tensor(CS, device="cuda", dtype=torch.float64, requires_grad=bool(case["turb"]))
        model, y = _Model(case, cs), x
        for _ in range(case["steps"]):
            y = model.step(y, recompute=True)
        wrt = list(x) + ([cs] if case["turb"] else [])
        return [a.detach() for a in y] + list(torch.autograd.grad(y, wrt,
                                                                  grad_outputs=[g.double() for g in _seeds(case, seed)]))
    with torch.no_grad():
        model = _Model(case)
        if kind == "corrected":
            ws, bs = _layers(_net(seed, 0.3))
            scale = _scale(_state(case, seed))
        for _ in range(case["steps"]):
            x = model.step(x)
            if kind == "corrected":
                x = _correct(x, ws, bs, scale)
    return list(x)
