"""The work a program gives this library, as cases that can be timed and
compared: the operators of a timestep one by one, whole timesteps and the
step's adjoint, each through fluid_simulator_backup_b200.Solver.

A case is a dict of plain values: `op` (the entry point), `precision` ("fp64"
or "fp32", the FP32 + FP64 refinement context), the grid `nx`, `ny`, `nz`
(dx = 1/nx) and the `scene` its level set and phases come from.  prepare()
makes the inputs in device memory and the solver that a program keeps, run()
is one pass: hand over what the operator overwrites, call it, take the results
back.  exact() restates the operators in plain FP64 torch."""
import math

import torch

import fluid_simulator_backup_b200 as fs

GRAVITY = (0.0, -9.8, 0.0)
EPS = 1e-6           # WENO5 epsilon
REINIT, SCALING = 10, 5
FACES = ("u", "v", "w")

# phases (phi <= 0 first): densities and viscosities
SCENES = {
    "bubble": dict(rho_neg=1.0, rho_pos=1000.0, mu_neg=1.8e-5, mu_pos=1e-3),   # air sphere in water
    "dam": dict(rho_neg=1000.0, rho_pos=1.0, mu_neg=1e-3, mu_pos=1.8e-5),      # water column in air
    "taylor": dict(rho_neg=850.0, rho_pos=1000.0, mu_neg=5e-2, mu_pos=1e-3),   # oil under water
}

# what each entry point overwrites (handed over on every pass) and returns
OPS = {
    "step": (("phi", "u", "v", "w", "pressure"), ("phi", "u", "v", "w", "pressure")),
    "step_adjoint": (("phi", "u", "v", "w", "pressure", "adj_phi", "adj_u", "adj_v", "adj_w"),
                     ("phi", "u", "v", "w", "adj_phi", "adj_u", "adj_v", "adj_w")),
    "project": (("u", "v", "w", "pressure"), ("u", "v", "w", "pressure")),
    "viscosity": (("u", "v", "w"), ("u", "v", "w")),
    "advect_levelset": (("phi",), ("phi",)),
    "advect_velocity": (("u", "v", "w"), ("u", "v", "w")),
    "reinitialize": (("phi",), ("phi",)),
}


def _case(name, op, precision, scene, nx, ny, nz, **more):
    return dict(name=name, op=op, precision=precision, scene=scene, nx=nx, ny=ny, nz=nz, **more)


def listed():
    return [
        # the production timestep: rising bubble at 256^3, FP32 fields, pressure to 1e-6 relative divergence
        _case("step_bubble_256", "step", "fp32", "bubble", 256, 256, 256, tolerance=1e-6),
        # the FP64 dam break at 64^3: the run others are checked against
        _case("step_dam_64_fp64", "step", "fp64", "dam", 64, 64, 64, tolerance=1e-8),
        # one backward step of the differentiable dam break (gradients by checkpointed rollout), 96^3
        _case("step_adjoint_dam_96", "step_adjoint", "fp32", "dam", 96, 96, 96, tolerance=1e-11),
        # the pressure projection alone on an ordinary, ragged box
        _case("project_bubble_150x210x131", "project", "fp32", "bubble", 150, 210, 131, tolerance=1e-6),
        # a small projection, where launches and latency count
        _case("project_dam_40", "project", "fp32", "dam", 40, 40, 40, tolerance=1e-6),
        # the plain FP64 projection
        _case("project_bubble_96_fp64", "project", "fp64", "bubble", 96, 96, 96, tolerance=1e-8),
        # level-set transport at full size
        _case("advect_levelset_256", "advect_levelset", "fp32", "bubble", 256, 256, 256),
        # velocity self-advection, WENO5, a ragged box
        _case("advect_velocity_200x136x267", "advect_velocity", "fp32", "dam", 200, 136, 267),
        # velocity self-advection with ENO3 (the scripts' scheme) in FP64, odd extents
        _case("advect_velocity_eno3_65x97x41_fp64", "advect_velocity", "fp64", "dam", 65, 97, 41, eno3=True),
        # one reinitialisation block at full size
        _case("reinitialize_256", "reinitialize", "fp32", "bubble", 256, 256, 256),
        # a small reinitialisation block in FP64
        _case("reinitialize_33x47x29_fp64", "reinitialize", "fp64", "bubble", 33, 47, 29),
        # semi-implicit viscosity of the oil/water instability
        _case("viscosity_taylor_128", "viscosity", "fp32", "taylor", 128, 128, 128),
    ]


# op -> precisions, scenes and the range of the mean extent
RANGES = {
    "step": (("fp32", "fp32", "fp64"), ("bubble", "dam", "taylor"), 24, 160),
    "step_adjoint": (("fp32", "fp64"), ("bubble", "dam"), 20, 80),
    "project": (("fp32", "fp32", "fp64"), ("bubble", "dam", "taylor"), 24, 200),
    "viscosity": (("fp32", "fp64"), ("taylor", "taylor", "bubble"), 24, 160),
    "advect_levelset": (("fp32", "fp64"), ("bubble", "dam", "taylor"), 24, 256),
    "advect_velocity": (("fp32", "fp64"), ("bubble", "dam", "taylor"), 24, 220),
    "reinitialize": (("fp32", "fp64"), ("bubble", "dam", "taylor"), 24, 256),
}


def draw(rng):
    op = rng.choice(sorted(RANGES))
    precisions, scenes, lo, hi = RANGES[op]
    precision = rng.choice(precisions)
    if precision == "fp64" and op in ("step", "step_adjoint", "project"):
        hi = 72 if op != "project" else 112
    mean = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = [max(17, round(mean * rng.uniform(0.75, 1.25))) for _ in range(3)]
    while n[0] * n[1] * n[2] > hi ** 3:
        n = [max(17, int(0.95 * a)) for a in n]
    c = dict(op=op, precision=precision, scene=rng.choice(scenes), nx=n[0], ny=n[1], nz=n[2])
    if op in ("step", "project"):
        c["tolerance"] = 1e-6 if precision == "fp32" else 1e-8
    if op == "step_adjoint":
        c["tolerance"] = 1e-11
    if op == "advect_velocity":
        c["eno3"] = rng.random() < 0.4
    return c


def work(case):
    """Bytes: every array handed over and taken back, once, as FP64 values (the
    interface's type).  Flops: the stencils of one pass, each solve counted as
    one application of its operator."""
    cells = case["nx"] * case["ny"] * case["nz"]
    up, down = OPS[case["op"]]
    weno = 3 * 110
    flops = {"advect_levelset": weno, "advect_velocity": 3 * weno, "reinitialize": REINIT * 2 * weno,
             "project": 60, "viscosity": 3 * 120}
    flops["step"] = 3 * (flops["advect_levelset"] + flops["advect_velocity"] + flops["reinitialize"] +
                         flops["project"] + flops["viscosity"])
    flops["step_adjoint"] = 3 * flops["step"]
    return {"bytes": 8.0 * cells * (len(up) + len(down)), "flops": float(cells * flops[case["op"]])}


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _axis(n, dx, face, dev):
    return (torch.arange(n + (1 if face else 0), dtype=torch.float64, device=dev) + (0.0 if face else 0.5)) * dx


def _distance(case, rnd, dev):
    """The scene's level set: a signed distance (negative in the first phase)
    whose gradient a past advection has stretched by up to 5 %."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = 1.0 / nx
    L = (1.0, ny * dx, nz * dx)
    x, y, z = (_axis(n, dx, False, dev) for n in (nx, ny, nz))
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    j = [0.04 * (q - 0.5) for q in rnd(5)]
    if case["scene"] == "bubble":
        r = (0.15 + 0.5 * j[0]) * min(L)
        phi = torch.sqrt((X - (0.5 + j[1]) * L[0]) ** 2 + (Y - (0.25 + j[2]) * L[1]) ** 2 + (Z - (0.5 + j[3]) * L[2]) ** 2) - r
    elif case["scene"] == "dam":
        dxw, dyw = X - (0.4 + j[0]) * L[0], Y - (0.6 + j[1]) * L[1]
        phi = torch.sqrt(dxw.clamp(min=0) ** 2 + dyw.clamp(min=0) ** 2) + torch.maximum(dxw, dyw).clamp(max=0)
        phi = phi.expand(nz, ny, nx)
    else:
        pert = torch.zeros(nz, nx, dtype=torch.float64, device=dev)
        q = rnd(4 * 6)
        for m in range(6):
            kx, kz = 1 + m % 3, 1 + m // 3
            pert += (q[4 * m] - 0.5) * torch.outer(torch.cos(2 * math.pi * (kz * z / L[2] + q[4 * m + 1])),
                                                   torch.cos(2 * math.pi * (kx * x / L[0] + q[4 * m + 2])))
        phi = (Y - (0.5 + j[0]) * L[1]) - 0.01 * pert[:, None, :] / pert.abs().max()
    q = [math.pi * a for a in rnd(3)]
    stretch = torch.cos(math.pi * X / L[0] + q[0]) * torch.cos(math.pi * Y / L[1] + q[1]) * torch.cos(math.pi * Z / L[2] + q[2])
    return phi * (1.0 + 0.05 * stretch)


def _velocity(case, rnd, dev):
    """A divergence-free MAC field that vanishes on the walls' normal faces:
    the discrete curl of a vector potential on the edges, peak 0.5."""
    n = (case["nx"], case["ny"], case["nz"])
    dx = 1.0 / n[0]

    def potential(axis):
        # on the edges along `axis`: cell centred there, face centred on the other two, zero on their walls
        total = 0.0
        q = rnd(5 * 4)
        for m in range(4):
            f = []
            for a in range(3):
                s = _axis(n[a], dx, a != axis, dev) / (n[a] * dx)
                k = 1 + int(3 * q[5 * m + a])
                f.append(torch.cos(math.pi * (k * s + q[5 * m + 3])) if a == axis else torch.sin(math.pi * k * s))
            total = total + (q[5 * m + 4] - 0.5) * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
        return total

    px, py, pz = potential(0), potential(1), potential(2)
    u = (pz[:, 1:, :] - pz[:, :-1, :]) - (py[1:] - py[:-1])
    v = (px[1:] - px[:-1]) - (pz[:, :, 1:] - pz[:, :, :-1])
    w = (py[:, :, 1:] - py[:, :, :-1]) - (px[:, 1:, :] - px[:, :-1, :])
    peak = torch.stack([a.abs().max() for a in (u, v, w)]).max()
    return [0.5 * a / peak for a in (u, v, w)]


def _dt(case):
    dx = 1.0 / case["nx"]
    return 0.5 * dx / (1.5 + math.sqrt(9.8 * dx))


def _inputs(case, seed):
    dev = _device()
    gen = torch.Generator().manual_seed(1 + seed)

    def rnd(k):
        return torch.rand(k, generator=gen, dtype=torch.float64).tolist()

    P = SCENES[case["scene"]]
    phi = _distance(case, rnd, dev)
    u, v, w = _velocity(case, rnd, dev)
    dx, dt = 1.0 / case["nx"], _dt(case)
    f = {"phi": phi, "u": u, "v": v, "w": w}
    if case["op"] == "project":
        # what the projection meets: the field after one advection and gravity
        for a, name in enumerate(FACES):
            g = f[name]
            ax = 2 - a
            k = [math.pi * (1 + q) for q in range(3)]
            s = [torch.arange(m, dtype=torch.float64, device=dev) / m for m in g.shape]
            mode = torch.cos(k[a] * s[0])[:, None, None] * torch.cos(k[(a + 1) % 3] * s[1])[None, :, None] * \
                torch.cos(k[(a + 2) % 3] * s[2])[None, None, :]
            g = g + 0.02 * mode + dt * GRAVITY[a]
            inner = torch.zeros_like(g)
            inner.narrow(ax, 1, g.shape[ax] - 2).copy_(g.narrow(ax, 1, g.shape[ax] - 2))
            f[name] = inner
    # the pressure of the step before: near hydrostatic
    rho = torch.where(phi <= 0, P["rho_neg"], P["rho_pos"]).to(torch.float64)
    column = -GRAVITY[1] * dx * rho
    f["pressure"] = column.flip(1).cumsum(1).flip(1) - 0.5 * column
    if case["op"] == "step_adjoint":
        # the bars of a mismatch with a target surface and of the kinetic energy
        y = _axis(case["ny"], dx, False, dev)[None, :, None]
        f["adj_phi"] = 2.0 * (phi - (y - 0.3))
        for name in FACES:
            f["adj_" + name] = 2.0 * f[name]
    up = OPS[case["op"]][0]
    if case["precision"] == "fp32":
        # an FP32 context's own values; its pressure and its bars are FP64
        for name in ("phi",) + FACES:
            f[name] = f[name].float().double()
    return {k: a.contiguous() for k, a in f.items() if k in up or k in ("phi",) + FACES}


def _params(case):
    p = dict(SCENES[case["scene"]], gravity=GRAVITY, weno_epsilon=EPS, reinit_iterations=REINIT,
             reinit_scaling=SCALING, order=3, stop=fs.FS_STOP_RELATIVE, max_iteration=40000,
             viscosity=1 if case["op"] in ("step", "step_adjoint", "viscosity") else 0,
             viscosity_tolerance=1e-12 if case["op"] == "step_adjoint" or case["precision"] == "fp64" else 1e-8,
             precision=fs.FS_PRECISION_FP64 if case["precision"] == "fp64" else fs.FS_PRECISION_FP32_REFINE)
    if "tolerance" in case:
        p["tolerance"] = case["tolerance"]
    if case.get("eno3"):
        p["velocity_scheme"] = fs.FS_VELOCITY_ENO3
    return p


def prepare(case, seed):
    up, down = OPS[case["op"]]
    fields = _inputs(case, seed)
    n = (case["nx"], case["ny"], case["nz"])
    solver = fs.Solver(n, 1.0 / n[0], **_params(case))
    torch.cuda.current_stream().synchronize()
    for name in ("phi",) + FACES:
        solver.upload_device(name, fields[name].data_ptr())
    out = {name: torch.empty(solver.shape(name), dtype=torch.float64, device=_device()) for name in down}
    if case["op"] == "step_adjoint":
        solver.adjoint_reset()
    return {"solver": solver, "op": case["op"], "dt": _dt(case), "in": {k: fields[k] for k in up}, "out": out,
            "fp32": case["precision"] == "fp32"}


def run(state):
    s, op, dt = state["solver"], state["op"], state["dt"]
    # the solver has a stream of its own: what this program queued on its stream has to be done first
    torch.cuda.current_stream().synchronize()
    if op == "step_adjoint":
        s.adjoint_reset()
    for name, a in state["in"].items():
        s.upload_device(name, a.data_ptr())
    if op == "step":
        s.step(dt)
    elif op == "step_adjoint":
        s.step_adjoint(dt)
    elif op == "project":
        s.project(dt)
    elif op == "viscosity":
        s.viscosity(dt)
    elif op == "advect_levelset":
        s.advect_levelset(dt)
    elif op == "advect_velocity":
        s.advect_velocity(dt)
    else:
        s.reinitialize()
    out = {}
    for name, a in state["out"].items():
        s.download_device(name, a.data_ptr())
        out[name] = a.float() if state["fp32"] else a  # an FP32 context's program goes on in FP32
    if op == "step_adjoint":
        out["rho_bars"] = torch.tensor(s.density_bars(), dtype=torch.float32 if state["fp32"] else torch.float64)
    return out


# ---------------------------------------------------------------- the operators in FP64


def _pad(f, ghosts, extrapolate):
    """Ghost layers on all sides, x first, then y, then z: linear
    extrapolation (level set) or zero (velocities)."""
    for ax in (2, 1, 0):
        n = f.shape[ax]
        lo, lo1, hi, hi1 = f.narrow(ax, 0, 1), f.narrow(ax, 1, 1), f.narrow(ax, n - 1, 1), f.narrow(ax, n - 2, 1)
        m = range(1, ghosts + 1)
        if extrapolate:
            below, above = [(q + 1) * lo - q * lo1 for q in reversed(m)], [(q + 1) * hi - q * hi1 for q in m]
        else:
            below = above = [torch.zeros_like(lo)] * ghosts
        f = torch.cat([*below, f, *above], ax)
    return f


def _samples(p, ax, shape):
    """The seven samples along an axis of an array padded by three."""
    out = []
    for o in range(7):
        q = p
        for a in range(3):
            q = q.narrow(a, o if a == ax else 3, shape[a])
        out.append(q)
    return out


def _weno(r1, r2, r3, r4, r5):
    s1 = 13 / 12 * (r1 - 2 * r2 + r3) ** 2 + 0.25 * (r1 - 4 * r2 + 3 * r3) ** 2
    s2 = 13 / 12 * (r2 - 2 * r3 + r4) ** 2 + 0.25 * (r2 - r4) ** 2
    s3 = 13 / 12 * (r3 - 2 * r4 + r5) ** 2 + 0.25 * (3 * r3 - 4 * r4 + r5) ** 2
    a1, a2, a3 = 0.1 / (EPS + s1) ** 2, 0.6 / (EPS + s2) ** 2, 0.3 / (EPS + s3) ** 2
    u1 = r1 / 3 - 7 / 6 * r2 + 11 / 6 * r3
    u2 = -r2 / 6 + 5 / 6 * r3 + r4 / 3
    u3 = r3 / 3 + 5 / 6 * r4 - r5 / 6
    return (a1 * u1 + a2 * u2 + a3 * u3) / (a1 + a2 + a3)


def _weno_sides(v, dx):
    d = [(b - a) / dx for a, b in zip(v, v[1:])]
    return _weno(*d[:5]), _weno(*d[:0:-1])


def _eno_sides(v, dx):
    d1 = [(b - a) / dx for a, b in zip(v, v[1:])]
    d2 = [(b - a) / (2 * dx) for a, b in zip(d1, d1[1:])]
    d3 = [(b - a) / (3 * dx) for a, b in zip(d2, d2[1:])]

    def pick(a, b):
        return torch.where(a.abs() <= b.abs(), a, b)

    h, h2 = dx, dx * dx
    dm = torch.where(d2[1].abs() <= d2[2].abs(), d1[2] + d2[1] * h + 2 * pick(d3[0], d3[1]) * h2,
                     d1[2] + d2[2] * h - pick(d3[1], d3[2]) * h2)
    dp = torch.where(d2[2].abs() <= d2[3].abs(), d1[3] - d2[2] * h - pick(d3[1], d3[2]) * h2,
                     d1[3] - d2[3] * h + 2 * pick(d3[2], d3[3]) * h2)
    return dm, dp


def _transport(f, vel, dt, dx, extrapolate, sides=_weno_sides):
    p = _pad(f, 3, extrapolate)
    out = f.clone()
    for a in range(3):
        dm, dp = sides(_samples(p, 2 - a, f.shape), dx)
        out -= dt * vel[a] * torch.where(vel[a] > 0, dm, dp)
    return out


def _mean2(f, ax):
    n = f.shape[ax]
    return 0.5 * (f.narrow(ax, 0, n - 1) + f.narrow(ax, 1, n - 1))


def _levelset(phi, vel, dt, dx):
    return _transport(phi, [_mean2(f, 2 - a) for a, f in enumerate(vel)], dt, dx, True)


def _advect(vel, dt, dx, sides=_weno_sides):
    out = []
    for a, f in enumerate(vel):
        at = []
        for b, g in enumerate(vel):
            if b == a:
                at.append(f)
            else:  # the mean of the four faces of component b around a face of component a
                g = _mean2(g, 2 - b)
                ax = 2 - a
                z = torch.zeros_like(g.narrow(ax, 0, 1))
                at.append(_mean2(torch.cat([z, g, z], ax), ax))
        out.append(_transport(f, at, dt, dx, False, sides))
    return out


def _reinitialize(phi, dx):
    s = phi / torch.sqrt(phi * phi + dx * dx)
    f = phi
    for _ in range(REINIT):
        p = _pad(f, 3, True)
        g2 = 0.0
        for a in range(3):
            dm, dp = _weno_sides(_samples(p, a, f.shape), dx)
            sm, sp = s * dm, s * dp
            shock = s * (dp.abs() - dm.abs()) / (dp - dm)
            g = torch.where((sp > 0) & (sm < 0), 0.0 * dm, torch.where(shock > 0, dm, dp))
            g = torch.where((sp <= 0) & (sm <= 0), dp, g)
            g = torch.where((sp >= 0) & (sm >= 0), dm, g)
            g2 = g2 + g * g
        r = f - dx / SCALING * s * (torch.sqrt(g2) - 1)
        f = torch.where(s * r < 0, EPS * torch.sign(s), r)
    return f


def _conjugate_gradients(apply, diag, b, x, tolerance):
    """Jacobi-preconditioned; the test every 20 iterations."""
    r = b - apply(x)
    bb = float((b * b).sum())
    if bb == 0.0:
        return torch.zeros_like(b)
    z = r / diag
    p, rz = z.clone(), (r * z).sum()
    for it in range(20000):
        if it % 20 == 0 and float((r * r).sum()) <= tolerance ** 2 * bb:
            break
        q = apply(p)
        alpha = rz / (p * q).sum()
        x = x + alpha * p
        r = r - alpha * q
        z = r / diag
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _divergence(vel, dx):
    return sum((f.narrow(2 - a, 1, f.shape[2 - a] - 1) - f.narrow(2 - a, 0, f.shape[2 - a] - 1)) / dx
               for a, f in enumerate(vel))


def _project(phi, vel, p, dt, dx, P):
    """The variable-density projection with the ghost-fluid face densities;
    the pressure is defined up to a constant."""
    inv = torch.where(phi <= 0, 1.0 / P["rho_neg"], 1.0 / P["rho_pos"]).to(torch.float64)
    beta = []
    for a in range(3):
        ax = 2 - a
        n = phi.shape[ax] - 1
        bc, bn = inv.narrow(ax, 1, n), inv.narrow(ax, 0, n)
        ac, an = phi.narrow(ax, 1, n).abs(), phi.narrow(ax, 0, n).abs()
        beta.append(bc * bn * (an + ac) / (bn * ac + bc * an))

    def apply(x):
        q = torch.zeros_like(x)
        for a in range(3):
            ax = 2 - a
            n = x.shape[ax] - 1
            flux = beta[a] * (x.narrow(ax, 1, n) - x.narrow(ax, 0, n)) / dx ** 2
            q.narrow(ax, 1, n).add_(flux)
            q.narrow(ax, 0, n).sub_(flux)
        return q

    diag = torch.zeros_like(phi)
    for a in range(3):
        n = phi.shape[2 - a] - 1
        diag.narrow(2 - a, 1, n).add_(beta[a] / dx ** 2)
        diag.narrow(2 - a, 0, n).add_(beta[a] / dx ** 2)
    b = -_divergence(vel, dx) / dt
    p = _conjugate_gradients(apply, diag, b - b.mean(), p, 1e-12)
    out = []
    for a, f in enumerate(vel):
        ax = 2 - a
        n = phi.shape[ax] - 1
        f = f.clone()
        f.narrow(ax, 1, n).sub_(dt * beta[a] * (p.narrow(ax, 1, n) - p.narrow(ax, 0, n)) / dx)
        out.append(f)
    return out, p


def _smeared(phi, e):
    h = 0.5 * (1 + phi / e + torch.sin(math.pi * phi / e) / math.pi)
    return torch.where(phi < -e, 0.0, torch.where(phi > e, 1.0, h))


def _viscosity(phi, vel, dt, dx, P, tolerance):
    """Semi-implicit: per component (rho_f - dt div mu grad) u = rho_f u* +
    the transposed stress, velocities zero beyond the walls."""
    e = 1.5 * dx
    pad = _pad(phi, 1, True)

    def mu(f):
        return P["mu_neg"] + (P["mu_pos"] - P["mu_neg"]) * _smeared(f, e)

    out = []
    for a, f in enumerate(vel):
        ax, shape = 2 - a, f.shape

        def cell(da, t=None, dt_=0):  # the cell on the low (da = -1) or high (0) side, shifted along t
            o = [1, 1, 1]
            o[ax] += da
            if t is not None:
                o[t] += dt_
            return pad[o[0]:o[0] + shape[0], o[1]:o[1] + shape[1], o[2]:o[2] + shape[2]]

        rho = P["rho_neg"] + (P["rho_pos"] - P["rho_neg"]) * _smeared(0.5 * (cell(-1) + cell(0)), e)
        low, high = [None] * 3, [None] * 3
        for d in range(3):
            if d == ax:
                low[d], high[d] = 2 * mu(cell(-1)), 2 * mu(cell(0))
            else:
                low[d] = mu(0.25 * (cell(-1, d, -1) + cell(-1) + cell(0, d, -1) + cell(0)))
                high[d] = mu(0.25 * (cell(-1) + cell(-1, d, 1) + cell(0) + cell(0, d, 1)))
        rhs = f.clone()
        for d in range(3):
            if d == ax:
                continue
            g = vel[2 - d]
            z = torch.zeros_like(g.narrow(ax, 0, 1))
            g = torch.cat([z, g, z], ax)
            jump = g.narrow(ax, 1, shape[ax]) - g.narrow(ax, 0, shape[ax])  # across the face, along the component's axis
            rhs = rhs + dt / rho * (high[d] * jump.narrow(d, 1, shape[d]) - low[d] * jump.narrow(d, 0, shape[d])) / dx ** 2
        inner = torch.zeros_like(f)
        inner.narrow(ax, 1, shape[ax] - 2).fill_(1.0)
        diag = torch.where(inner > 0, rho + dt / dx ** 2 * sum(low[d] + high[d] for d in range(3)), 1.0)

        def apply(x):
            p = _pad(x, 1, False)
            q = diag * x
            for d in range(3):
                up, dn = [1, 1, 1], [1, 1, 1]
                up[d], dn[d] = 2, 0
                hi = p[up[0]:up[0] + shape[0], up[1]:up[1] + shape[1], up[2]:up[2] + shape[2]]
                lo = p[dn[0]:dn[0] + shape[0], dn[1]:dn[1] + shape[1], dn[2]:dn[2] + shape[2]]
                q = q - dt / dx ** 2 * inner * (high[d] * hi + low[d] * lo)
            return torch.where(inner > 0, q, x)

        out.append(_conjugate_gradients(apply, diag, rho * rhs * inner, f * inner, tolerance))
    return out


def _step(phi, vel, p, dt, dx, P, tolerance):
    f1 = _levelset(phi, vel, dt, dx)
    f2 = 0.75 * phi + 0.25 * _levelset(f1, vel, dt, dx)
    new = phi / 3 + 2 / 3 * _levelset(f2, vel, dt, dx)
    cur = vel
    for c0, c1 in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
        cur = _advect(cur, dt, dx)
        for a, f in enumerate(cur):
            f.narrow(2 - a, 0, 1).zero_()
            f.narrow(2 - a, f.shape[2 - a] - 1, 1).zero_()
            f.narrow(2 - a, 1, f.shape[2 - a] - 2).add_(dt * GRAVITY[a])
        cur = _viscosity(new, cur, dt, dx, P, tolerance)
        cur, p = _project(new, cur, p, dt, dx, P)
        cur = [c0 * f0 + c1 * f for f0, f in zip(vel, cur)]
    f1 = _reinitialize(new, dx)
    f2 = 0.75 * new + 0.25 * _reinitialize(f1, dx)
    return new / 3 + 2 / 3 * _reinitialize(f2, dx), cur


def exact(case, seed):
    op = case["op"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if op == "step_adjoint" or (op == "step" and cells > 3_000_000):
        return None
    f = _inputs(case, seed)
    phi, vel = f["phi"], [f[k] for k in FACES]
    dx, dt, P = 1.0 / case["nx"], _dt(case), SCENES[case["scene"]]
    if op == "advect_levelset":
        return {"phi": _levelset(phi, vel, dt, dx)}
    if op == "reinitialize":
        return {"phi": _reinitialize(phi, dx)}
    if op == "advect_velocity":
        return dict(zip(FACES, _advect(vel, dt, dx, _eno_sides if case.get("eno3") else _weno_sides)))
    if op == "viscosity":
        return dict(zip(FACES, _viscosity(phi, vel, dt, dx, P, 1e-13)))
    if op == "project":
        vel, _ = _project(phi, vel, f["pressure"], dt, dx, P)
        return dict(zip(FACES, vel), pressure=None)
    phi, vel = _step(phi, vel, f["pressure"], dt, dx, P, 1e-13)
    return dict(zip(FACES, vel), phi=phi, pressure=None)
