"""
Performance cases: the calls a program that runs circumbinary disks with this
package makes, over the range of sizes and options it makes them in.

A case is a dict of plain values with a "kind":

  step     one driver iteration of the isothermal solver through the host
           loop: dt from maximum_wavespeed(), advance(dt), reductions()
  run      the device-resident driver loop, Solver.run(steps)
  kernels  the four drop-in kernels through the C-ABI on the caller's arrays
  gamma    one driver iteration of the gamma-law solver
  batch    many disks in one launch, BatchedSolver.run(steps), and their states
  adjoint  a run and the gradient of its mean accretion rate and torque

prepare() builds the inputs on the device from the seed (a disk with a few
spiral modes and zone noise) and the solver a program keeps; run() is one pass
through the public calls; exact() is the same result in plain torch float64.
"""

import ctypes
import math

import numpy as np
import torch

THETA = 1.5
MODELS = {"acceleration_free": 1, "torque_free": 2, "force_free": 3}
BATCH_SIZES = (128, 192, 256, 384, 512, 768, 1024)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest grid that is stepped from the host: launches, host work
        # and the read of the wavespeed
        dict(name="step_64", kind="step", setup="disk", n=64, radius=8.0, rk=2, q=1.0, e=0.0),
        # the code-comparison disk at its default resolution, third order, with
        # its own six diagnostics (more than the stage's epilogue holds)
        dict(name="step_kitp_200", kind="step", setup="kitp", n=200, radius=8.0, rk=3, q=1.0, e=0.0),
        # an odd size, default domain (spacing not a power of two), eccentric binary
        dict(name="step_1511", kind="step", setup="disk", n=1511, radius=12.0, rk=2, q=0.4, e=0.3),
        # the throughput grid
        dict(name="step_4096", kind="step", setup="disk", n=4096, radius=8.0, rk=2, q=1.0, e=0.0),
        # the device loop on an ordinary grid, whole graphs of steps
        dict(name="run_1024", kind="run", n=1024, radius=8.0, steps=16, precision="exact", q=1.0, e=0.0),
        # the device loop in the fast arithmetic, a group shorter than a graph
        dict(name="run_2048_fast", kind="run", n=2048, radius=8.0, steps=4, precision="fast", q=0.7, e=0.1),
        # a program that binds the four kernels itself
        dict(name="kernels_1000", kind="kernels", n=1000, radius=8.0, q=1.0, e=0.2),
        # the gamma-law disk at the setup's default resolution
        dict(name="gamma_512", kind="gamma", n=512, radius=12.0, cooling=0.0, follow=False, mdots=False, q=1.0, e=0.0),
        # an odd size with cooling, softening that follows the disk height, accretion rates every step
        dict(name="gamma_cool_1153", kind="gamma", n=1153, radius=6.0, cooling=1.0, follow=True, mdots=True, q=0.5, e=0.2),
        # the gamma-law throughput grid
        dict(name="gamma_2048", kind="gamma", n=2048, radius=12.0, cooling=0.0, follow=False, mdots=False, q=1.0, e=0.0),
        # a parameter study: disks of many sizes, and their states at the end
        dict(name="batch_24", kind="batch", disks=24, largest=1024, steps=16),
        # a gradient with checkpoints
        dict(name="adjoint_512", kind="adjoint", n=512, steps=40, every=20, store=False),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "run", "run", "kernels", "gamma", "gamma", "gamma", "batch", "adjoint"])
    q, e = round(rng.uniform(0.1, 1.0), 3), rng.choice([0.0, round(rng.uniform(0.0, 0.5), 3)])
    radius = rng.choice([8.0, 12.0, round(rng.uniform(5.0, 15.0), 2)])
    if kind == "step":
        setup = rng.choice(["disk", "disk", "kitp"])
        n = _log_size(rng, 48, 4096 if setup == "disk" else 640)
        return dict(kind=kind, setup=setup, n=n, radius=radius, rk=rng.choice([1, 2, 2, 2, 3]), q=q, e=e)
    if kind == "run":
        n = _log_size(rng, 64, 2048)
        return dict(kind=kind, n=n, radius=radius, steps=rng.randint(2, 24),
                    precision=rng.choice(["exact", "exact", "fma", "fast"]), q=q, e=e)
    if kind == "kernels":
        return dict(kind=kind, n=_log_size(rng, 100, 2048), radius=radius, q=q, e=e)
    if kind == "gamma":
        return dict(kind=kind, n=_log_size(rng, 64, 2048), radius=radius, cooling=rng.choice([0.0, 0.5]),
                    follow=rng.choice([False, False, True]), mdots=rng.choice([False, True]), q=q, e=e)
    if kind == "batch":
        return dict(kind=kind, disks=rng.randint(3, 24), largest=rng.choice([256, 512, 1024]),
                    steps=rng.randint(4, 16))
    return dict(kind=kind, n=_log_size(rng, 128, 512), steps=rng.randint(8, 40), every=rng.choice([8, 20]),
                store=rng.choice([False, True]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centres(n, radius):
    d = 2.0 * radius / n
    c = -radius + (torch.arange(n, dtype=torch.float64, device=_device()) + 0.5) * d
    return c[:, None], c[None, :]


def _kitp_sigma(r):
    return 1e-5 + (1.0 - 1e-5) * math.exp(-((2.5 / r) ** 12))


def _state(setup, n, radius, seed):
    """Primitive zones (n, n, 3 or 4): the setup's disk, spiral modes in
    Sigma and the radial velocity, 1e-3 noise."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    x, y = _centres(n, radius)
    r = torch.sqrt(x * x + y * y)
    rs = torch.sqrt(x * x + y * y + 0.05 ** 2)
    phi = torch.atan2(y.expand(n, n), x.expand(n, n))
    modes = torch.rand(3, 3, generator=g, device=dev, dtype=torch.float64)

    def noise(size):
        return 1.0 + size * (2.0 * torch.rand(n, n, generator=g, device=dev, dtype=torch.float64) - 1.0)

    swirl = torch.zeros(n, n, dtype=torch.float64, device=dev)
    for m in range(3):
        a, wind, phase = modes[m, 0] * 0.05, 2.0 + 3.0 * modes[m, 1], 6.28 * modes[m, 2]
        swirl += a * torch.cos((m + 1) * phi + wind * torch.log(rs) + phase)
    del phi
    vphi = torch.sqrt(1.0 / rs)
    if setup == "kitp":
        sigma = 1e-5 + (1.0 - 1e-5) * torch.exp(-((2.5 / r) ** 12))
        omega0 = torch.sqrt(0.99 / r ** 3)
        vphi = r * (omega0 ** -4 + 1.0) ** -0.25
        fields = [sigma]
    elif setup == "gamma":
        taper = 0.0001 + 0.9999 * torch.exp(-((1.0 / rs) ** 30))
        fields = [rs ** -0.6 * taper, 1e-2 * rs ** -1.5 * taper]
    else:
        fields = [torch.ones_like(rs)]
    vr = 0.1 * vphi * swirl
    rc = torch.clamp(r, min=1e-12)
    out = [fields[0] * (1.0 + swirl) * noise(1e-3), (vr * x - vphi * y) / rc, (vr * y + vphi * x) / rc]
    if setup == "gamma":
        out.append(fields[1] * (1.0 + swirl) * noise(1e-3))
    return torch.stack(out, dim=-1).contiguous()


def _on_host(state):
    from sailfish_b200 import pinned_empty

    host = pinned_empty(tuple(state.shape))
    torch.from_numpy(host).copy_(state)
    return host


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

DIAGNOSTICS = [dict(quantity="time"), dict(quantity="mdot", which_mass=1, accretion=True),
               dict(quantity="mdot", which_mass=2, accretion=True),
               dict(quantity="torque", which_mass="both", gravity=True)]


def _setup(case):
    from sailfish_b200.setups import CircumbinaryDisk, KitpCodeComparison

    common = dict(domain_radius=case["radius"], mass_ratio=case["q"], eccentricity=case["e"])
    if case.get("setup") == "kitp":
        return KitpCodeComparison(**common)
    if case["kind"] == "gamma":
        return CircumbinaryDisk(eos="gamma-law", cooling_coefficient=case["cooling"],
                                constant_softening=not case["follow"],
                                which_diagnostics="mdots" if case["mdots"] else "none", **common)
    return CircumbinaryDisk(**common)


def _batch(case, seed):
    """(n, q, e, mach, nu) of every disk of a batch: sizes in turn, parameters over the study's ranges."""
    rng = np.random.default_rng(seed)
    sizes = [s for s in BATCH_SIZES if s <= case["largest"]]
    out = []
    for i in range(case["disks"]):
        out.append((sizes[i % len(sizes)], float(rng.uniform(0.1, 1.0)), float(rng.uniform(0.0, 0.5)),
                    float(rng.uniform(10.0, 40.0)), float(10.0 ** rng.uniform(-4.0, -2.0))))
    return out


def _mass_args(m):
    return [m.position_x, m.position_y, m.velocity_x, m.velocity_y, m.mass, m.softening_length, m.sink_rate,
            m.sink_radius, m.sink_model.value]


def prepare(case, seed):
    from sailfish_b200 import make_solver

    kind = case["kind"]
    if kind in ("step", "run", "gamma"):
        setup = _setup(case)
        mesh = setup.mesh(case["n"])
        physics = setup.physics
        options = dict(plm_theta=THETA)
        if kind != "gamma":
            options.update(rk_order=case.get("rk", 2), precision=case.get("precision", "exact"))
            if case.get("setup") != "kitp":
                physics["diagnostics"] = DIAGNOSTICS
        name = "gamma" if kind == "gamma" else case.get("setup", "disk")
        solver = make_solver(setup.solver, physics, options, setup=setup, mesh=mesh,
                             solution=_on_host(_state(name, case["n"], case["radius"], seed)))
        return dict(case=case, solver=solver, mesh=mesh)
    if kind == "kernels":
        from sailfish_b200 import _capi

        setup = _setup(case)
        mesh = setup.mesh(case["n"])
        n, r = case["n"], case["radius"]
        lib = _capi.lib()
        padded = torch.zeros(n + 4, n + 4, 3, dtype=torch.float64, device="cuda")
        padded[2:-2, 2:-2] = _state("disk", n, r, seed)
        _fill_guards(padded)
        arrays = dict(prim=padded, cons=torch.zeros_like(padded), out=padded.clone(),
                      speed=torch.zeros(n + 4, n + 4, dtype=torch.float64, device="cuda"),
                      rate=torch.zeros_like(padded))
        masses = [_mass_args(m) for m in setup.point_masses(0.3)]
        return dict(case=case, lib=lib, mesh=mesh, masses=masses, **arrays)
    if kind == "batch":
        from sailfish_b200.batched import BatchedSolver, Disk
        from sailfish_b200.setups import CircumbinaryDisk

        disks = []
        for i, (n, q, e, mach, nu) in enumerate(_batch(case, seed)):
            setup = CircumbinaryDisk(domain_radius=8.0, mach_number=mach, mass_ratio=q, eccentricity=e, nu=nu)
            disks.append(Disk(setup, setup.mesh(n), _on_host(_state("disk", n, 8.0, seed * 100 + i))))
        return dict(case=case, solver=BatchedSolver(disks, plm_theta=THETA, diagnostics=DIAGNOSTICS[1:]))
    if kind == "adjoint":
        from sailfish_b200.adjoint import AdjointRun, Params

        run_ = AdjointRun(resolution=case["n"], steps=case["steps"], checkpoint_every=case["every"],
                          store_states=case["store"])
        return dict(case=case, run=run_, params=Params(), prim=_on_host(_state("disk", case["n"], 8.0, seed)))
    raise ValueError(kind)


def _fill_guards(a):
    """The caller's outflow boundary: two zero-gradient zones on every side."""
    a[:2], a[-2:] = a[2:3].clone(), a[-3:-2].clone()
    a[:, :2], a[:, -2:] = a[:, 2:3].clone(), a[:, -3:-2].clone()


def _row(values):
    return np.array(values, dtype=complex if any(isinstance(v, complex) for v in values) else float)


def _interior(solver):
    return solver.state_buffer()[2:-2, 2:-2]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "gamma"):
        s = state["solver"]
        dt = state["mesh"].min_spacing() / s.maximum_wavespeed() * s.recommended_cfl
        s.advance(dt)
        return dict(dt=dt, series=_row(s.reductions()), prim=_interior(s))
    if kind == "run":
        s = state["solver"]
        return dict(series=np.array(s.run(case["steps"])), prim=_interior(s))
    if kind == "kernels":
        return _run_kernels(state)
    if kind == "batch":
        b = state["solver"]
        series = b.run(case["steps"])
        return dict(series=[np.array(rows) for rows in series], prim=[b.solution(i) for i in range(case["disks"])])
    r = state["run"]
    value = r.forward(state["prim"], state["params"], keep=True)
    grad_state, grad_params = r.gradient((1.0, 0.5))
    return dict(value=value, state=grad_state, params=grad_params)


def _run_kernels(state):
    """The drop-in kernels as a solver that binds them calls them in one RK
    stage: conserved state, stage, wavespeeds, one mass's source rates."""
    lib, mesh, n = state["lib"], state["mesh"], state["case"]["n"]
    r = state["case"]["radius"]
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    lib.cbdiso_b200_set_plm_theta(THETA)
    prim, cons, out, speed, rate = (ctypes.c_void_p(state[k].data_ptr()) for k in
                                    ("prim", "cons", "out", "speed", "rate"))
    m1, m2 = state["masses"]
    edges = (-r, r, -r, r)
    status = lib.cbdiso_2d_primitive_to_conserved(n, n, prim, cons)
    status |= lib.cbdiso_2d_advance_rk(n, n, *edges, cons, prim, out, 1.0, 1.0, 100.0, r, 1.0, 1, *m1, *m2, 0.0,
                                       100.0, 2, 1e-3, 0.0, 0.05 * mesh.dx, 1e12, 1e-12)
    status |= lib.cbdiso_2d_wavespeed(n, n, *edges, 0.0, 100.0, 2, *m1, *m2, out, speed)
    status |= lib.cbdiso_2d_point_mass_source_term(n, n, *edges, *m1, out, rate)
    if status:
        raise RuntimeError(f"drop-in kernel status {status}")
    return dict(cons=state["cons"][2:-2, 2:-2], prim=state["out"][2:-2, 2:-2], speed=state["speed"][2:-2, 2:-2],
                rate=state["rate"][2:-2, 2:-2])


def work(case):
    """Bytes: each stage reads the state (and, beyond the first, u_n) and
    writes it, float64; operations: the float64 ones of a stage's arithmetic
    that any form has (slopes, face fluxes, sources, recovery), per zone."""
    kind = case["kind"]
    stages, extra = {1: (1, 48), 2: (2, 120), 3: (3, 192)}[case.get("rk", 2)]
    flops = 400.0 * stages
    if kind == "step":
        zones = case["n"] ** 2
    elif kind == "run":
        zones = case["n"] ** 2 * case["steps"]
    elif kind == "kernels":
        zones, extra, flops = case["n"] ** 2, 24 + 24 + 24 + 24 + 8 + 24, 480.0
    elif kind == "gamma":
        zones, extra, flops = case["n"] ** 2, 160, 1600.0
    elif kind == "batch":
        zones = sum(d[0] ** 2 for d in _batch(case, 0)) * case["steps"]
    else:
        # forward, and backward with about twice its traffic and operations
        zones, extra, flops = case["n"] ** 2 * case["steps"], 3 * 120, 3 * 800.0
    return dict(bytes=float(zones * extra), flops=float(zones * flops))


# ---------------------------------------------------------------------------
# the same results in plain torch, float64 (fields first: [q, i, j])
# ---------------------------------------------------------------------------


def _kepler(t, q, e):
    """Both bodies' (x, y, vx, vy, mass) at time t for a = M = 1, as tensors
    differentiable in q and e."""
    n = t - 2.0 * math.pi * math.floor(t / (2.0 * math.pi))
    k, e0 = n, float(e.detach())
    for _ in range(50):
        k = k - (k - e0 * math.sin(k) - n) / (1.0 - e0 * math.cos(k))
    k = torch.as_tensor(k, dtype=torch.float64)
    k = k - (k - e * torch.sin(k) - n) / (1.0 - e * torch.cos(k))
    ck, sk, b = torch.cos(k), torch.sin(k), torch.sqrt(1.0 - e * e)
    f = q / (1.0 + q)
    x, y = f * (ck - e), f * sk * b
    w = 1.0 / (1.0 - e * ck)
    vx, vy = -f * w * sk, f * w * ck * b
    m1 = 1.0 / (1.0 + q)
    return [(x, y, vx, vy, m1), (-x / q, -y / q, -vx / q, -vy / q, 1.0 - m1)]


def _pad(p):
    p = torch.cat([p[:, :1], p[:, :1], p, p[:, -1:], p[:, -1:]], dim=1)
    return torch.cat([p[:, :, :1], p[:, :, :1], p, p[:, :, -1:], p[:, :, -1:]], dim=2)


def _minmod(a, b, c):
    l, m, r = (b - a) * THETA, (c - a) * 0.5, (c - b) * THETA
    least = torch.minimum(l.abs(), torch.minimum(m.abs(), r.abs()))
    same = (torch.sign(l) == torch.sign(m)) & (torch.sign(l) == torch.sign(r))
    return torch.where(same, torch.sign(m) * least, torch.zeros_like(least))


def _slopes(p):
    c = p[:, 1:-1, 1:-1]
    return c, _minmod(p[:, :-2, 1:-1], c, p[:, 2:, 1:-1]), _minmod(p[:, 1:-1, :-2], c, p[:, 1:-1, 2:])


class _Grid:
    def __init__(self, n, radius, dev):
        self.n, self.d, self.radius = n, 2.0 * radius / n, radius
        k = torch.arange(n + 1, dtype=torch.float64, device=dev)
        self.f, self.c = -radius + k * self.d, -radius + (k[:-1] + 0.5) * self.d
        self.x, self.y = self.c[:, None], self.c[None, :]


def _sink(m, cfg, dx, dy):
    """Sink rate of one mass and the distance to it."""
    r = torch.sqrt(dx * dx + dy * dy)
    s = cfg["rate"] * torch.exp(-((r / 0.05) ** 4))
    return torch.where(r < 0.2, s, torch.zeros_like(s)), r


def _sink_velocity(m, model, dx, dy, r, vx, vy):
    if model == 1:
        return vx, vy
    if model == 3:
        return torch.zeros_like(vx), torch.zeros_like(vy)
    ex, ey = dx / (r + 1e-12), dy / (r + 1e-12)
    v = (vx - m[2]) * ex + (vy - m[3]) * ey
    return v * ex + m[2], v * ey + m[3]


def _gravity(m, dx, dy, soft2):
    return -m[4] * (dx * dx + dy * dy + soft2) ** -1.5


def _iso_cs2(masses, cfg, x, y):
    phi = sum(m[4] / torch.sqrt((x - m[0]) ** 2 + (y - m[1]) ** 2 + 0.05 ** 2) for m in masses)
    return phi / cfg["mach"] ** 2


def _hlle(ul, ur, fl, fr, vl, vr, cs):
    am = torch.clamp(torch.minimum(vl, vr) - cs, max=0.0)
    ap = torch.clamp(torch.maximum(vl, vr) + cs, min=0.0)
    return (fl * ap - fr * am - (ul - ur) * ap * am) / (ap - am)


def _iso_face(pl, pr, cs2, axis):
    def cons_flux(p):
        u = torch.stack([p[0], p[0] * p[1], p[0] * p[2]])
        f = u * p[1 + axis]
        press = p[0] * cs2
        return u, torch.stack([f[0], f[1] + press if axis == 0 else f[1], f[2] + press if axis == 1 else f[2]])

    (ul, fl), (ur, fr) = cons_flux(pl), cons_flux(pr)
    return _hlle(ul, ur, fl, fr, pl[1 + axis], pr[1 + axis], torch.sqrt(cs2))


def _iso_strain(c, gx, gy, d):
    sxx, syy = (4.0 * gx[1] - 2.0 * gy[2]) / (3.0 * d), (4.0 * gy[2] - 2.0 * gx[1]) / (3.0 * d)
    return c[0] * sxx, c[0] * (gx[2] + gy[1]) / d, c[0] * syy


def _iso_stage(p, un, g, cfg, masses, a, dt):
    """One RK stage of primitive zones p; un the conserved zones of the step's start."""
    c, gx, gy = _slopes(_pad(p))
    sxx, sxy, syy = _iso_strain(c, gx, gy, g.d)
    i = slice(1, -1)
    half = 0.5 * cfg["nu"]
    fx = _iso_face((c + 0.5 * gx)[:, :-1, i], (c - 0.5 * gx)[:, 1:, i], _iso_cs2(masses, cfg, g.f[:, None], g.y), 0)
    zero = torch.zeros_like(fx[0])
    fx = fx - half * torch.stack([zero, sxx[:-1, i] + sxx[1:, i], sxy[:-1, i] + sxy[1:, i]])
    fy = _iso_face((c + 0.5 * gy)[:, i, :-1], (c - 0.5 * gy)[:, i, 1:], _iso_cs2(masses, cfg, g.x, g.f[None, :]), 1)
    zero = torch.zeros_like(fy[0])
    fy = fy - half * torch.stack([zero, sxy[i, :-1] + sxy[i, 1:], syy[i, :-1] + syy[i, 1:]])
    u = torch.stack([p[0], p[0] * p[1], p[0] * p[2]])
    du = torch.zeros_like(u)
    r = torch.clamp(torch.sqrt(g.x ** 2 + g.y ** 2), min=1e-12)
    onset = g.radius - 1.0
    if cfg["buffer"] is not None:
        sb = cfg["buffer"]
        vk = torch.sqrt(1.0 / r)
        rate = torch.clamp(r - onset, min=0.0) * 100.0 * math.sqrt(onset ** -3.0)
        target = torch.stack([sb + 0.0 * r, -sb * g.y / r * vk, sb * g.x / r * vk])
        du = du - (u - target) * rate * dt
    for m in masses:
        dx, dy = g.x - m[0], g.y - m[1]
        acc = p[0] * _gravity(m, dx, dy, 0.05 ** 2) * dt
        s, dist = _sink(m, cfg, dx, dy)
        vx, vy = _sink_velocity(m, cfg["model"], dx, dy, dist, p[1], p[2])
        loss = -dt * s * p[0]
        du = du + torch.stack([loss, loss * vx + acc * dx, loss * vy + acc * dy])
    du = du - (fx[:, 1:] - fx[:, :-1] + fy[:, :, 1:] - fy[:, :, :-1]) / g.d * dt
    u = (1.0 - a) * (u + du) + a * un
    rho = torch.clamp(u[0], min=1e-12)
    return torch.stack([rho, u[1] / rho, u[2] / rho])


def _iso_speed(p, g, cfg, masses):
    cs = torch.sqrt(_iso_cs2(masses, cfg, g.x, g.y))
    return torch.maximum(p[1].abs() + cs, p[2].abs() + cs)


def _iso_sums(p, g, cfg, masses):
    """(mdot 1, mdot 2, torque on both) sums times the zone area."""
    out, torque = [], 0.0
    for m in masses:
        dx, dy = g.x - m[0], g.y - m[1]
        out.append(-(_sink(m, cfg, dx, dy)[0] * p[0]).sum() * g.d ** 2)
        f = p[0] * _gravity(m, dx, dy, 0.05 ** 2)
        torque = torque + f * (g.x * dy - g.y * dx)
    return out, torque


def _iso_row(p, g, cfg, masses, time, kitp):
    mdots, torque = _iso_sums(p, g, cfg, masses)
    d2 = g.d ** 2
    row = [time / (2.0 * math.pi)] + [float(v) for v in mdots] + [float(torque.sum() * d2)]
    if kitp:
        r = torch.sqrt(g.x ** 2 + g.y ** 2)
        row.append(float((torque * ((r > 1.0) & (r < g.radius))).sum() * d2))
        row.append(complex((p[0] * g.x / r).sum(), (p[0] * g.y / r).sum()) * d2)
        s = p[0] * ((r > 1.0) & (r < 6.0))
        vv, vr = p[1] ** 2 + p[2] ** 2, p[1] * g.x + p[2] * g.y
        row.append(complex((s * (vv * g.x - vr * p[1] - g.x / r)).sum(),
                           (s * (vv * g.y - vr * p[2] - g.y / r)).sum()) * d2)
    return row


RK = {1: (0.0,), 2: (0.0, 0.5), 3: (0.0, 0.75, 1.0 / 3.0)}


def _iso_step(p, g, cfg, time, dt, rk, q, e):
    un = torch.stack([p[0], p[0] * p[1], p[0] * p[2]])
    t = time
    for a in RK[rk]:
        p = _iso_stage(p, un, g, cfg, _kepler(t, q, e), a, dt)
        t = time * a + (t + dt) * (1.0 - a)
    return p, t


def _iso_config(case):
    kitp = case.get("setup") == "kitp"
    onset = case.get("radius", 8.0) - 1.0
    return dict(mach=10.0, nu=1e-3, rate=10.0, model=1 if kitp else 2, buffer=_kitp_sigma(onset) if kitp else 1.0)


def _tensor(v):
    return torch.tensor(float(v), dtype=torch.float64)


def _exact_iso(prim, n, radius, cfg, q, e, rk, steps, kitp=False):
    """(dts, rows, final zones) of a driver run."""
    g = _Grid(n, radius, prim.device)
    p, t, q, e = prim.permute(2, 0, 1), 0.0, _tensor(q), _tensor(e)
    dts, rows = [], []
    for _ in range(steps):
        dt = g.d / float(_iso_speed(p, g, cfg, _kepler(t, q, e)).max()) * 0.3
        p, t = _iso_step(p, g, cfg, t, dt, rk, q, e)
        dts.append(dt)
        rows.append(_iso_row(p, g, cfg, _kepler(t, q, e), t, kitp))
    return dts, rows, p.permute(1, 2, 0)


def _gam_stage(p, un, g, cfg, masses, a, dt):
    gam, alpha = 5.0 / 3.0, 0.1
    c, gx, gy = _slopes(_pad(p))
    i = slice(1, -1)
    temp = c[3] / c[0]
    cs, sq = torch.sqrt(temp * gam), torch.sqrt(temp)
    sxx, syy = (4.0 * gx[1] - 2.0 * gy[2]) / (3.0 * g.d), (4.0 * gy[2] - 2.0 * gx[1]) / (3.0 * g.d)
    sxy = (gx[2] + gy[1]) / g.d

    def height(x, y):
        return torch.sqrt(sum(m[4] * ((x - m[0]) ** 2 + (y - m[1]) ** 2 + 1e-12) ** -1.5 for m in masses))

    def cons(v):
        return torch.stack([v[0], v[0] * v[1], v[0] * v[2], v[3] / (gam - 1.0) + 0.5 * v[0] * (v[1] ** 2 + v[2] ** 2)])

    def faces(lo, hi, axis):
        """Both sides' states and fluxes of the faces along an axis."""
        sides = []
        for v in (lo, hi):
            u = cons(v)
            f = u * v[1 + axis]
            f = torch.stack([f[0], f[1] + v[3] if axis == 0 else f[1], f[2] + v[3] if axis == 1 else f[2],
                             f[3] + v[3] * v[1 + axis]])
            sides.append((u, f, v[1 + axis]))
        return sides

    def viscous(z, nu, axis):
        """Stress flux of a zone's own strain with viscosity nu."""
        s1, s2 = (z["sxx"], z["sxy"]) if axis == 0 else (z["sxy"], z["syy"])
        w = nu * z["rho"]
        return torch.stack([torch.zeros_like(w), w * s1, w * s2, w * s1 * z["vx"] + w * s2 * z["vy"]])

    def zones(si, sj):
        return dict(sxx=sxx[si, sj], sxy=sxy[si, sj], syy=syy[si, sj], rho=c[0][si, sj], vx=c[1][si, sj],
                    vy=c[2][si, sj])

    here = zones(i, i)
    hc = sq[i, i] / height(g.x, g.y)
    nuc = alpha * hc * cs[i, i]
    div = 0.0
    lo, hi = slice(0, -2), slice(2, None)
    for axis in (0, 1):
        if axis == 0:
            left, right = (c + 0.5 * gx)[:, :-1, i], (c - 0.5 * gx)[:, 1:, i]
            w = height(g.f[:, None], g.y)
            cut = lambda f, k: f[..., k, :]  # noqa: E731
            near = ((lo, i), (hi, i))
        else:
            left, right = (c + 0.5 * gy)[:, i, :-1], (c - 0.5 * gy)[:, i, 1:]
            w = height(g.x, g.f[None, :])
            cut = lambda f, k: f[..., k]  # noqa: E731
            near = ((i, lo), (i, hi))
        (ul, fl, vl), (ur, fr, vr) = faces(left, right, axis)
        for sign, side, at in ((-1.0, slice(None, -1), near[0]), (1.0, slice(1, None), near[1])):
            # each face of a zone takes the neighbour's sound speed and height
            f = _hlle(*(cut(v, side) for v in (ul, ur, fl, fr, vl, vr)), cs[at])
            nun = alpha * sq[at] / cut(w, side) * cs[at]
            f = f - 0.5 * (viscous(zones(*at), nun, axis) + viscous(here, nuc, axis))
            div = div + sign * f / g.d
    u = cons(p)
    r = torch.clamp(torch.sqrt(g.x ** 2 + g.y ** 2), min=1e-12)
    onset = g.radius - 0.1
    rate = torch.clamp(r - onset, min=0.0) / 0.1 * 1000.0 * math.sqrt(onset ** -3.0)
    sb, pb = cfg["sigma"], cfg["pressure"]
    vk = torch.sqrt(1.0 / r)
    target = torch.stack([sb + 0.0 * r, -sb * vk * g.y / r, sb * vk * g.x / r, pb / (gam - 1.0) + 0.5 * sb * vk ** 2])
    u = u - (u - target) * rate * dt
    eps = p[3] / p[0] / (gam - 1.0)
    for m in masses:
        dx, dy = g.x - m[0], g.y - m[1]
        s, dist = _sink(m, cfg, dx, dy)
        soft = 0.05
        if cfg["follow"]:
            b = (1.0 - (dist / 0.05) ** 2) ** 2
            soft = torch.where(dist > 0.05, 0.5 * hc, b * 0.05 + (1.0 - b) * 0.5 * hc)
        acc = p[0] * _gravity(m, dx, dy, soft ** 2) * dt
        vx, vy = _sink_velocity(m, 2, dx, dy, dist, p[1], p[2])
        loss = -dt * s * p[0]
        u = u + torch.stack([loss, loss * vx + acc * dx, loss * vy + acc * dy,
                             loss * (eps + 0.5 * (vx ** 2 + vy ** 2)) + acc * (dx * p[1] + dy * p[2])])
    cooled = eps * (1.0 + 3.0 * cfg["cooling"] * p[0] ** -2 * eps ** 3 * dt) ** (-1.0 / 3.0)
    cooled = torch.maximum(cooled, (p[1] ** 2 + p[2] ** 2) / gam / (gam - 1.0) * 1e-10)
    u = torch.cat([u[:3], (u[3] + p[0] * (cooled - eps))[None]])
    u = (1.0 - a) * (u - div * dt) + a * un
    pres = torch.clamp((u[3] - 0.5 * (u[1] ** 2 + u[2] ** 2) / u[0]) * (gam - 1.0), min=1e-12)
    out = torch.stack([u[0], u[1] / u[0], u[2] / u[0], pres])
    floor = torch.tensor([1e-10, 0.0, 0.0, 1e-12], dtype=torch.float64, device=p.device)[:, None, None]
    return torch.where(u[0] < 1e-10, floor, out)


def _exact_gamma(case, seed):
    prim = _state("gamma", case["n"], case["radius"], seed)
    g = _Grid(case["n"], case["radius"], prim.device)
    q, e = _tensor(case["q"]), _tensor(case["e"])
    rs = math.sqrt((case["radius"] - 0.1) ** 2 + 0.05 ** 2)
    taper = 0.0001 + 0.9999 * math.exp(-((1.0 / rs) ** 30))
    cfg = dict(rate=10.0, sigma=rs ** -0.6 * taper, pressure=1e-2 * rs ** -1.5 * taper, cooling=case["cooling"],
               follow=case["follow"])
    p = prim.permute(2, 0, 1)
    cs = torch.sqrt(p[3] / p[0] * 5.0 / 3.0)
    dt = g.d / float(torch.maximum(p[1].abs() + cs, p[2].abs() + cs).max()) * 0.1
    un = torch.stack([p[0], p[0] * p[1], p[0] * p[2], p[3] * 1.5 + 0.5 * p[0] * (p[1] ** 2 + p[2] ** 2)])
    p = _gam_stage(p, un, g, cfg, _kepler(0.0, q, e), 0.0, dt)
    p = _gam_stage(p, un, g, cfg, _kepler(dt, q, e), 0.5, dt)
    row = []
    if case["mdots"]:
        row = [dt / (2.0 * math.pi)] + [float(-(_sink(m, cfg, g.x - m[0], g.y - m[1])[0] * p[0]).sum() * g.d ** 2)
                                        for m in _kepler(dt, q, e)]
    return dict(dt=dt, series=_row(row), prim=p.permute(1, 2, 0))


def _exact_kernels(case, seed):
    n, radius = case["n"], case["radius"]
    prim = _state("disk", n, radius, seed)
    g = _Grid(n, radius, prim.device)
    cfg = _iso_config(case)
    masses = _kepler(0.3, _tensor(case["q"]), _tensor(case["e"]))
    p = prim.permute(2, 0, 1)
    cons = torch.stack([p[0], p[0] * p[1], p[0] * p[2]])
    out = _iso_stage(p, cons, g, cfg, masses, 0.0, 0.05 * g.d)
    m = masses[0]
    dx, dy = g.x - m[0], g.y - m[1]
    s, dist = _sink(m, cfg, dx, dy)
    vx, vy = _sink_velocity(m, 2, dx, dy, dist, out[1], out[2])
    loss, acc = -s * out[0], out[0] * _gravity(m, dx, dy, 0.05 ** 2)
    rate = torch.stack([loss, loss * vx + acc * dx, loss * vy + acc * dy])
    return dict(cons=cons.permute(1, 2, 0), prim=out.permute(1, 2, 0), speed=_iso_speed(out, g, cfg, masses),
                rate=rate.permute(1, 2, 0))


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    n = case["n"]
    prim = _state("disk", n, 8.0, seed)
    g = _Grid(n, 8.0, prim.device)
    prim = prim.permute(2, 0, 1).contiguous().requires_grad_(True)
    par = [_tensor(v).requires_grad_(True) for v in (0.5, 0.1, 1e-3, 10.0)]  # q, e, nu, sink rate

    def step(p, t, dt, q, e, nu, rate):
        cfg = dict(mach=10.0, nu=nu, rate=rate, model=2, buffer=1.0)
        p, end = _iso_step(p, g, cfg, t, dt, 2, q, e)
        mdots, torque = _iso_sums(p, g, cfg, _kepler(end, q, e))
        return p, -(mdots[0] + mdots[1]) * dt, torque.sum() * g.d ** 2 * dt

    p, t, total, mdot, torque = prim, 0.0, 0.0, 0.0, 0.0
    for _ in range(case["steps"]):
        with torch.no_grad():
            cfg = dict(mach=10.0)
            dt = g.d / float(_iso_speed(p, g, cfg, _kepler(t, par[0], par[1])).max()) * 0.3
        p, a, b = checkpoint(step, p, t, dt, *par, use_reentrant=False)
        mdot, torque, total = mdot + a, torque + b, total + dt
        t = t * 0.5 + (t + dt + dt) * 0.5
    value = torch.stack([mdot, torque]) / total
    grads = torch.autograd.grad(value[0] + 0.5 * value[1], [prim] + par)
    return dict(value=value.detach().cpu().numpy(), state=grads[0].permute(1, 2, 0).contiguous().cpu().numpy(),
                params=np.array([float(v) for v in grads[1:]]))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "run"):
        kitp = case.get("setup") == "kitp"
        prim = _state(case.get("setup", "disk"), case["n"], case["radius"], seed)
        steps = case.get("steps", 1)
        dts, rows, p = _exact_iso(prim, case["n"], case["radius"], _iso_config(case), case["q"], case["e"],
                                  case.get("rk", 2), steps, kitp)
        if kind == "step":
            return dict(dt=dts[0], series=_row(rows[0]), prim=p)
        return dict(series=np.array([row + [dt] for row, dt in zip(rows, dts)]), prim=p)
    if kind == "kernels":
        return _exact_kernels(case, seed)
    if kind == "gamma":
        return _exact_gamma(case, seed)
    if kind == "batch":
        series, prims = [], []
        for i, (n, q, e, mach, nu) in enumerate(_batch(case, seed)):
            cfg = dict(mach=mach, nu=nu, rate=10.0, model=2, buffer=1.0)
            dts, rows, p = _exact_iso(_state("disk", n, 8.0, seed * 100 + i), n, 8.0, cfg, q, e, 2, case["steps"])
            series.append(np.array([row[1:] + [dt] for row, dt in zip(rows, dts)]))
            prims.append(p.cpu().numpy())
        return dict(series=series, prim=prims)
    return _exact_adjoint(case, seed)
