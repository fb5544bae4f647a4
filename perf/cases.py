"""Timed cases of the per-timestep hot path.

Every case goes through cajitafluids_gb300.Context as a program does: host
arrays of the owned regions go in, whole steps run on the device, host arrays
come out.  Inputs are seeded: a spectral streamfunction velocity (rms 1) and a
smooth scalar in [0, 1], the fields of the benchmark workloads.

Three forms:
  steps      upload q, u, v; Context.steps(n); download q, u, v: the solve loop
             between two output times (n steps with one synchronisation)
  step_host  Context.step_host: one step with host buffers in and out, as a
             host code that owns its fields calls it
  adjoint    upload; forward_checkpointed; backward from dL/dq, dL/du, dL/dv:
             one gradient of a loss on the final state

exact() restates a step in 64 bits with plain torch: RK3 trace and B-spline
samples by gathers, the projection by a direct (FFT) Poisson solve, and the
reverse sweep by automatic differentiation of those.
"""
from __future__ import annotations

import math

import torch

from cajitafluids_gb300 import Context, SolverOptions
from cajitafluids_gb300 import _lib as L

HALO = 3
DENSITY = 0.1  # the reference driver's default
# inflow block of the smoke and scalar-transport problems: location, size,
# velocity, quantity
INFLOW = ((0.45, 0.10), (0.10, 0.05), (0.0, 3.0), 1.0)
RATE = ((0.45, 0.10), (0.10, 0.05), (0.0, 0.0), 1.0)
GRAVITY = -9.8
MG_NAMES = ("PFMG", "SMG", "MG")


def _case(name, form, nx, ny, **kw):
    c = {"name": name, "form": form, "nx": nx, "ny": ny, "periodic": False, "precision": "fp64", "order": 3,
         "solver": "PCG", "precon": "PFMG", "tol": 1e-8, "abs_tol": 0.0, "inner_tol": 0.0, "steps": 1, "every": 0,
         "source": "none", "buoyancy": False, "fix_q1": True}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest grid a user debugs on, with the solver the reference's
        # own class defaults to (diagonal, 1e-6): launch and wait latencies
        _case("smoke 64 fp64 Reference", "steps", 64, 64, solver="Reference", precon="Diagonal", tol=1e-6, steps=4,
              source="inflow", fix_q1=False),
        # the plain method's standard problem: 256^2, walls, inflow, linear
        # values, Jacobi-PCG to 1e-8
        _case("inflow 256 fp64 Jacobi linear", "steps", 256, 256, order=1, precon="Diagonal", steps=3,
              source="inflow", fix_q1=False),
        # its larger form: cubic values, gravity scaled by the quantity, 1e-10
        _case("buoyancy 1024 fp64 Jacobi", "steps", 1024, 1024, precon="Diagonal", tol=1e-10, source="inflow",
              buoyancy=True, fix_q1=False),
        # an odd, non-square domain in mixed precision with the diagonal
        # preconditioner (odd extents do not coarsen)
        _case("ragged 501x333 mixed Jacobi", "steps", 501, 333, precision="mixed", precon="Diagonal", tol=1e-10,
              source="inflow", steps=2),
        # the command line's default solver pair on a small non-square domain
        _case("cli 192x160 fp64 PFMG", "steps", 192, 160, tol=1e-6, steps=10, source="inflow"),
        # a mid-size production run in mixed precision, walls and inflow
        _case("inflow 1024 mixed PFMG", "steps", 1024, 1024, precision="mixed", steps=10, source="inflow",
              inner_tol=0.5),
        # the headline workload: 4096^2 periodic, mixed, ||div u|| <= 1e-8
        _case("spectral 4096 mixed PFMG", "steps", 4096, 4096, periodic=True, precision="mixed", tol=0.0,
              abs_tol=1e-8, inner_tol=0.5, steps=8),
        # the same problem in plain FP64
        _case("spectral 4096 fp64 PFMG", "steps", 4096, 4096, periodic=True, tol=0.0, abs_tol=1e-8, steps=2),
        # the same step with host buffers in and out every step
        _case("host step 4096 mixed PFMG", "step_host", 4096, 4096, periodic=True, precision="mixed", tol=0.0,
              abs_tol=1e-8, inner_tol=0.5),
        # the largest grid: 8192^2 walls, mixed
        _case("spectral 8192 mixed PFMG", "steps", 8192, 8192, precision="mixed", tol=0.0, abs_tol=1e-8,
              inner_tol=0.5, steps=4),
        # gradient of a scalar-transport loss: 512^2, FP64, inflow rate
        _case("adjoint 512 fp64 PFMG", "adjoint", 512, 512, tol=1e-10, steps=6, every=3, source="rate"),
        # a large gradient in mixed precision
        _case("adjoint 4096 mixed PFMG", "adjoint", 4096, 4096, precision="mixed", tol=0.0, abs_tol=1e-8,
              inner_tol=0.5, steps=6, every=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: Jacobi or multigrid forward runs, or a gradient, over
    the sizes, axes, orders, precisions and inputs of the listed ones."""
    kind = rng.choice(("jacobi", "mg", "mg", "mg", "host", "adjoint"))
    precision = rng.choice(("fp64", "mixed"))
    periodic = rng.random() < 0.5
    order = rng.choice((1, 3, 3))
    source = rng.choice(("none", "inflow"))
    buoyancy = rng.random() < 0.25
    nx = _log_int(rng, 48, {"jacobi": 900, "mg": 4096, "host": 4096, "adjoint": 3000}[kind])
    ny = max(33, int(nx * rng.uniform(0.5, 1.0)))
    if precision == "fp64" and kind == "adjoint":
        nx, ny = min(nx, 700), min(ny, 700)
    if kind != "jacobi":
        # grids that coarsen: multiples of a power of two, an odd factor over it
        m = rng.choice((8, 16, 32)) if min(nx, ny) > 128 else 8
        nx, ny = max(48, nx // m * m), max(40, ny // m * m)
    cells = nx * ny
    c = _case("", {"jacobi": "steps", "mg": "steps", "host": "step_host", "adjoint": "adjoint"}[kind], nx, ny,
              periodic=periodic, precision=precision, order=order, source=source, buoyancy=buoyancy)
    del c["name"]
    if kind == "jacobi":
        c.update(precon="Diagonal", tol=1e-10 if precision == "mixed" else rng.choice((1e-6, 1e-8)),
                 fix_q1=precision == "mixed", steps=1 if cells > 100000 else 2)
    else:
        # updates after every iteration lower the FP32 form's attainable residual
        inner = rng.choice((0.0, 0.5)) if precision == "mixed" else 0.0
        c.update(tol=1e-8 if inner else rng.choice((1e-8, 1e-10)), inner_tol=inner)
    if kind == "mg":
        c["steps"] = max(1, min(8, (1 << 23) // cells))
    if kind == "adjoint":
        c.update(source=rng.choice(("none", "rate")), buoyancy=False, steps=rng.choice((2, 3, 4)), every=2)
    return c


# --------------------------------------------------------------------------
# inputs


def _spectral(ny, nx, slope, kmax, gen):
    """A real field on ny x nx points of one period: Gaussian coefficients,
    power |k|^slope for 1 <= |k| <= kmax."""
    dev = "cuda"
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64)
    kx = torch.arange(nx // 2 + 1, dtype=torch.float64)
    sy = torch.nonzero(ky.abs() <= kmax).ravel()
    sx = torch.nonzero(kx <= kmax).ravel()
    k = torch.sqrt(ky[sy][:, None] ** 2 + kx[sx][None, :] ** 2)
    amp = torch.where((k >= 1.0) & (k <= kmax), k.clamp(min=1.0) ** (slope / 2.0), torch.zeros_like(k))
    coef = torch.complex(torch.randn(k.shape, generator=gen, dtype=torch.float64) * amp,
                         torch.randn(k.shape, generator=gen, dtype=torch.float64) * amp)
    spec = torch.zeros((ny, nx // 2 + 1), dtype=torch.complex128, device=dev)
    spec[sy.to(dev)[:, None], sx.to(dev)[None, :]] = coef.to(dev)
    return torch.fft.irfft2(spec, s=(ny, nx))


def _fields(case, seed):
    """q, u, v (float64 tensors on the GPU, owned regions) and dt."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    nx, ny = case["nx"], case["ny"]
    dx = 1.0 / nx
    kmax = min(64, nx // 4, ny // 4)
    psi = _spectral(ny, nx, -11.0 / 3.0 - 2.0, kmax, gen)
    psi = torch.cat([psi, psi[:1]], 0)
    psi = torch.cat([psi, psi[:, :1]], 1)  # nodes
    if not case["periodic"]:
        wx = torch.sin(math.pi * torch.arange(nx + 1, device="cuda", dtype=torch.float64) / nx)
        wy = torch.sin(math.pi * torch.arange(ny + 1, device="cuda", dtype=torch.float64) / ny)
        psi = psi * wx[None, :] * wy[:, None]
        psi[0] = psi[-1] = 0.0
        psi[:, 0] = psi[:, -1] = 0.0
    u = (psi[1:] - psi[:-1]) / dx
    v = -(psi[:, 1:] - psi[:, :-1]) / dx
    if case["periodic"]:
        u, v = u[:, :-1], v[:-1]
    rms = torch.sqrt((u * u).mean() + (v * v).mean())
    u, v = (u / rms).contiguous(), (v / rms).contiguous()
    q = _spectral(ny, nx, -3.0, kmax, gen)
    q = ((q - q.min()) / (q.max() - q.min())).contiguous()
    top = max(float(u.abs().max()), float(v.abs().max()))
    if case["source"] == "inflow":
        top = max(top, abs(INFLOW[2][1]))
    return q, u, v, 0.5 * dx / top


def _seeds(case, seed, shapes):
    """dL/dq, dL/du, dL/dv of the final state (a smooth misfit plus noise)."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 31 + 5)
    return [torch.randn(s, generator=gen, device="cuda", dtype=torch.float64) for s in shapes]


def _pinned(shape, values=None):
    """A page-locked float64 array (the view keeps its memory alive)."""
    t = torch.empty(tuple(shape), dtype=torch.float64, pin_memory=True)
    if values is not None:
        t.copy_(values)
    return t.numpy()


def _options(case):
    return SolverOptions(solver=case["solver"], precon=case["precon"], tol=case["tol"], abs_tol=case["abs_tol"],
                         max_iter=100000, inner_tol=case["inner_tol"])


def prepare(case, seed):
    nx, ny = case["nx"], case["ny"]
    q, u, v, dt = _fields(case, seed)
    c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny * (1.0 / nx)), periodic=(case["periodic"],) * 2,
                precision=case["precision"])
    c.set_density(DENSITY)
    if case["fix_q1"]:
        c.set_quirks(L.CF_FIX_Q1)
    if case["source"] == "inflow":
        c.set_source(*INFLOW, mode=0)
    elif case["source"] == "rate":
        c.set_source(*RATE, mode=1)
    if case["buoyancy"]:
        c.set_body_force((0.0, GRAVITY), True)
    s = {"case": case, "ctx": c, "dt": dt, "opts": _options(case), "in": [_pinned(t.shape, t) for t in (q, u, v)]}
    if case["form"] == "adjoint":
        s["bar"] = [_pinned(t.shape, t) for t in _seeds(case, seed, (q.shape, u.shape, v.shape))]
    else:
        s["out"] = [_pinned(t.shape) for t in (q, u, v)]
    return s


def run(state):
    case, c, dt, opts = state["case"], state["ctx"], state["dt"], state["opts"]
    if case["form"] == "step_host":
        c.step_host(dt, case["order"], opts, *state["in"], *state["out"])
        return dict(zip("quv", state["out"]))
    for f, a in zip("quv", state["in"]):
        c.upload(f, a)
    if case["form"] == "adjoint":
        c.forward_checkpointed(case["steps"], case["every"], dt, case["order"], opts)
        return c.backward(*state["bar"])
    c.steps(case["steps"], dt, case["order"], opts)
    return {f: c.download(f, a) for f, a in zip("quv", state["out"])}


def work(case):
    """Bytes: the three fields in and out once (the adjoint: the final state's
    three adjoints in and three gradients out besides).  Operations: per step
    and cell about 300 for the three traces and samples of the advection (250
    more and twice that in reverse), 40 for divergence, gradient and norms, and
    the solver's count at its usual number of iterations (Jacobi: 13 each, about
    2.3 per cell along the longer axis; multigrid: 60 each, 8 of them)."""
    cells = case["nx"] * case["ny"]
    solve = 60.0 * 8 if case["precon"] in MG_NAMES else 13.0 * 2.3 * max(case["nx"], case["ny"])
    step = (300.0 if case["order"] == 3 else 200.0) + 40.0 + solve
    if case["form"] == "adjoint":
        return {"bytes": 72.0 * cells, "flops": case["steps"] * (2.0 * step + 500.0 + solve) * cells}
    return {"bytes": 48.0 * cells, "flops": case["steps"] * step * cells}


# --------------------------------------------------------------------------
# the same in 64 bits, without the library

OFF = {"q": (0.5, 0.5), "u": (0.0, 0.5), "v": (0.5, 0.0)}


class _Grid:
    """Rows [row0, row0 + len) of a ghosted field of extents (ey, ex)."""

    def __init__(self, t, row0, ex, ey):
        self.t, self.row0, self.ex, self.ey = t, row0, ex, ey


def _ghosted(f, kind, case):
    nx, ny = case["nx"], case["ny"]
    ex, ey = nx + 6 + (kind == "u"), ny + 6 + (kind == "v")
    if case["periodic"]:
        iy = (torch.arange(ey, device=f.device) - HALO) % ny
        ix = (torch.arange(ex, device=f.device) - HALO) % nx
        return f[iy][:, ix]
    return torch.nn.functional.pad(f, (HALO, ex - HALO - f.shape[1], HALO, ey - HALO - f.shape[0]))


def _weights(x, ext, order):
    if order == 1:
        x = x.clamp(0.0, float(ext - 1))
        k = x.detach().floor().clamp(max=float(ext - 2))
        t = x - k
        return k.long(), (1.0 - t, t)
    x = x.clamp(1.0, float(ext - 2))
    k = x.detach().floor().clamp(max=float(ext - 3))
    t = x - k
    s = 1.0 - t
    return k.long() - 1, (s ** 3 / 6.0, 0.5 * t ** 3 - t * t + 2.0 / 3.0, 0.5 * (t + t * t - t ** 3) + 1.0 / 6.0,
                          t ** 3 / 6.0)


def _sample(g, order, x, y):
    """g at index coordinates (x, y)."""
    kx, wx = _weights(x, g.ex, order)
    ky, wy = _weights(y, g.ey, order)
    flat = g.t.reshape(-1)
    base = (ky - g.row0) * g.ex + kx
    val = 0.0
    for b, wb in enumerate(wy):
        row = 0.0
        for a, wa in enumerate(wx):
            row = row + wa * flat[base + (b * g.ex + a)]
        val = val + wb * row
    return val


def _advected(kind, G, case, dt, j0, j1):
    """Advected values of the kind's entities in owned rows [j0, j1)."""
    nx = case["nx"]
    c = dt * nx
    cols = nx + (kind == "u" and not case["periodic"])
    dev = G["u"].t.device
    X = (torch.arange(cols, device=dev, dtype=torch.float64) + HALO + OFF[kind][0])[None, :]
    Y = (torch.arange(j0, j1, device=dev, dtype=torch.float64) + HALO + OFF[kind][1])[:, None]
    X, Y = X.expand(j1 - j0, cols), Y.expand(j1 - j0, cols)

    def vel(dx, dy):
        return (_sample(G["u"], 1, X + dx - OFF["u"][0], Y + dy - OFF["u"][1]),
                _sample(G["v"], 1, X + dx - OFF["v"][0], Y + dy - OFF["v"][1]))
    zero = torch.zeros_like(X)
    a = vel(zero, zero)
    b = vel(-0.5 * c * a[0], -0.5 * c * a[1])
    d = vel(-0.75 * c * a[0], -0.75 * c * a[1])
    fx, fy = [-c * ((2.0 / 9.0) * a[k] + (3.0 / 9.0) * b[k] + (4.0 / 9.0) * d[k]) for k in (0, 1)]
    return _sample(G[kind], case["order"], X + fx - OFF[kind][0], Y + fy - OFF[kind][1])


def _in_box(kind, shape, case, j0=0):
    (x0, y0), (w, h) = INFLOW[0], INFLOW[1]
    dx = 1.0 / case["nx"]
    x = (torch.arange(shape[1], device="cuda", dtype=torch.float64) + OFF[kind][0]) * dx
    y = (torch.arange(j0, j0 + shape[0], device="cuda", dtype=torch.float64) + OFF[kind][1]) * dx
    return ((y >= y0) & (y < y0 + h))[:, None] & ((x >= x0) & (x < x0 + w))[None, :]


def _inputs(q, u, v, case, dt, rate):
    if case["source"] == "inflow":
        q = torch.where(_in_box("q", q.shape, case), q.clamp(min=INFLOW[3]), q)
        # (the inflow velocity's x component is zero: no u is smaller)
        v = torch.where(_in_box("v", v.shape, case) & (v.abs() < INFLOW[2][1]), torch.full_like(v, INFLOW[2][1]), v)
    elif case["source"] == "rate":
        q = q + _in_box("q", q.shape, case) * (rate * dt)
    if case["buoyancy"]:
        if case["periodic"]:
            rho = 0.5 * (q + q.roll(1, 0))
        else:
            z = torch.zeros_like(q[:1])
            rho = 0.5 * (torch.cat([z, q]) + torch.cat([q, z]))
        v = v + dt * GRAVITY * rho
    if not case["periodic"]:
        u, v = _walls(u, v)
    return q, u, v


def _walls(u, v):
    u = torch.nn.functional.pad(u[:, 1:-1], (1, 1))
    v = torch.nn.functional.pad(v[1:-1], (0, 0, 1, 1))
    return u, v


def _poisson(b, scale, periodic):
    """x with A x = b, A = scale (4 x - neighbours): periodic, or reflecting
    walls (by even extension), mean zero."""
    ny, nx = b.shape
    if not periodic:
        b = torch.cat([b, b.flip(1)], 1)
        b = torch.cat([b, b.flip(0)], 0)
    my, mx = b.shape
    ly = 2.0 - 2.0 * torch.cos(2.0 * math.pi * torch.arange(my, device=b.device, dtype=torch.float64) / my)
    lx = 2.0 - 2.0 * torch.cos(2.0 * math.pi * torch.arange(mx // 2 + 1, device=b.device, dtype=torch.float64) / mx)
    lam = scale * (ly[:, None] + lx[None, :])
    lam[0, 0] = math.inf
    x = torch.fft.irfft2(torch.fft.rfft2(b) / lam, s=(my, mx))
    return x[:ny, :nx]


def _project(u, v, case, dt):
    nx, ny = case["nx"], case["ny"]
    dx = 1.0 / nx
    if case["periodic"]:
        div = (u.roll(-1, 1) - u) + (v.roll(-1, 0) - v)
    else:
        div = (u[:, 1:] - u[:, :-1]) + (v[1:] - v[:-1])
    p = _poisson(div / -dx, dt / (DENSITY * dx * dx), case["periodic"])
    s = dt / (DENSITY * dx)
    if case["periodic"]:
        return u - s * (p - p.roll(1, 1)), v - s * (p - p.roll(1, 0))
    if not case["fix_q1"]:
        # the unfixed wall rule leaves p in the wall rows of v, so the
        # pressure's constant matters: conjugate gradients with the diagonal
        # preconditioner keep the diagonal-weighted mean at zero
        d = torch.full_like(p, 4.0)
        d[0] -= 1.0
        d[-1] -= 1.0
        d[:, 0] -= 1.0
        d[:, -1] -= 1.0
        p = p - (d * p).sum() / d.sum()
    pad = torch.nn.functional.pad(p, (1, 1, 1, 1))
    u = u - s * (pad[1:-1, 1:] - pad[1:-1, :-1])
    v = v - s * (pad[1:, 1:-1] - pad[:-1, 1:-1])
    if case["fix_q1"]:
        return _walls(u, v)
    u = torch.nn.functional.pad(u[1:, 1:-1], (1, 1, 1, 0))
    return u, v


def _forward_advect(s, case, dt):
    G = {k: _Grid(_ghosted(f, k, case), 0, case["nx"] + 6 + (k == "u"), case["ny"] + 6 + (k == "v"))
         for k, f in zip("quv", s)}
    return [torch.cat([_advected(k, G, case, dt, j, min(j + 1024, f.shape[0])) for j in range(0, f.shape[0], 1024)])
            for k, f in zip("quv", s)]


def _reverse_advect(s, bars, case, dt):
    """Adjoint of _forward_advect at s, in row blocks."""
    ghosted = [_ghosted(f, k, case) for k, f in zip("quv", s)]
    total = [torch.zeros_like(g) for g in ghosted]
    rows = max(32, (1 << 21) // case["nx"])
    for kind, bar in zip("quv", bars):
        for j0 in range(0, bar.shape[0], rows):
            j1 = min(j0 + rows, bar.shape[0])
            G, at = {}, []
            for k, g in zip("quv", ghosted):
                a, b = max(0, j0 + HALO - 4), min(g.shape[0], j1 + HALO + 5)
                G[k] = _Grid(g[a:b].clone().requires_grad_(True), a, g.shape[1], g.shape[0])
                at.append((a, b))
            val = _advected(kind, G, case, dt, j0, j1)
            grads = torch.autograd.grad(val, [G[k].t for k in "quv"], bar[j0:j1], allow_unused=True)
            for t, g, (a, b) in zip(total, grads, at):
                if g is not None:
                    t[a:b] += g
    out = []
    for k, f, t in zip("quv", s, total):
        leaf = torch.zeros_like(f, requires_grad=True)
        out.append(torch.autograd.grad(_ghosted(leaf, k, case), leaf, t)[0])
    return out


def exact(case, seed):
    s = list(_fields(case, seed))
    dt = s.pop()
    steps = case["steps"]
    states = []
    for _ in range(steps):
        states.append(s)
        s = list(_inputs(*_forward_advect(s, case, dt), case, dt, RATE[3]))
        s[1:] = _project(s[1], s[2], case, dt)
    if case["form"] != "adjoint":
        return {k: f.cpu().numpy() for k, f in zip("quv", s)}
    bars = _seeds(case, seed, [f.shape for f in s])
    rate = 0.0
    for s in reversed(states):
        adv = [f.requires_grad_(True) for f in _forward_advect(s, case, dt)]
        r = torch.tensor(RATE[3], dtype=torch.float64, device="cuda", requires_grad=True)
        q, u, v = _inputs(*adv, case, dt, r)
        u, v = _project(u, v, case, dt)
        g = torch.autograd.grad([q, u, v], adv + [r], bars, allow_unused=True)
        rate += float(g[3]) if g[3] is not None else 0.0
        bars = _reverse_advect(s, g[:3], case, dt)
    out = {k: f.cpu().numpy() for k, f in zip("quv", bars)}
    out["rate"] = rate
    return out
