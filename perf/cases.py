"""The work that programs built on this package have it do, as cases that can be
timed and checked: the fractional step in its forms (FP64 and FP32 storage with
defect correction, central and upwind3 + RK2 advection, with and without the
sphere), the Poisson solve, spectral forcing, the diagnostics and the two
adjoints, through the public Python API on torch's current stream.

A case is a dict of plain values: ``kind`` (what the program calls, see
``listed``), the grid ``nx, ny, nz`` (powers of two in [16, 256]; FP32 storage
from nx = 32), ``precision``, ``scheme`` and ``steps`` per pass.

``exact`` restates each path in plain FP64 torch (rolls and torch.fft).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

import cubismup_3d_b200 as cup
from cubismup_3d_b200 import _lib as L
from cubismup_3d_b200 import adjoint

DEV = "cuda:0"
RADIUS, CENTRE = 0.1, (0.5, 0.5, 0.5)  # the sphere, in a box of longest side 2
EPS = 2.220446049250313080847e-16

# kinds with the sphere, and the steps a state has behind it before the first pass
SPHERE_KINDS = ("sphere", "moving", "obstacle_grad")
SPIN_UP = {"step": 2, "run": 4, "sphere": 40, "forced": 4, "obstacle_grad": 20, "diagnostics": 3}


def case(kind, cells, precision, scheme, steps, name=None):
    c = {"kind": kind, "nx": cells[0], "ny": cells[1], "nz": cells[2], "precision": precision, "scheme": scheme,
         "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    up = "upwind3_rk2"
    return [
        # the smallest call: one step of the reference's loop (calcMaxTimestep, timestep with its
        # stats on the host) on a coarse, elongated grid
        case("step", (32, 16, 64), "fp64", "ref", 1, "step_32x16x64_fp64_ref"),
        # Taylor-Green at 64^3, 50 steps from its initial condition: a whole small run
        case("short_run", (64, 64, 64), "fp64", up, 50, "taylor_green_64_fp64"),
        # the reference's loop with per-step stats on a ragged grid of ordinary size
        case("step", (128, 64, 256), "fp32_dc", up, 8, "step_128x64x256_fp32dc"),
        # decaying turbulence at 256^3, a long run in both precisions
        case("run", (256, 256, 256), "fp32_dc", up, 12, "turbulence_256_fp32dc"),
        case("run", (256, 256, 256), "fp64", up, 12, "turbulence_256_fp64"),
        # flow past the fixed sphere (fixed frame, implicit penalization), a long run
        case("sphere", (256, 128, 128), "fp32_dc", up, 12, "sphere_256x128x128_fp32dc"),
        # a sphere moving through the frame, the pipeline driven operator by operator
        case("moving", (128, 64, 64), "fp64", "ref", 8, "moving_sphere_128x64x64_fp64"),
        # gradient of a rollout with checkpoints every 8 steps (forward, recompute, backward)
        case("rollout_grad", (128, 128, 128), "fp32_dc", up, 16, "rollout_grad_128_fp32dc"),
        # gradient of the time-averaged drag with respect to u0, chi and the sphere's velocity
        case("obstacle_grad", (256, 128, 128), "fp32_dc", up, 4, "obstacle_grad_256x128x128_fp32dc"),
        # the periodic Poisson solver on its own
        case("poisson", (256, 256, 256), "fp64", "ref", 1, "poisson_256_fp64"),
        # homogeneous isotropic turbulence held at its energy by spectral forcing
        case("forced", (128, 128, 128), "fp32_dc", up, 6, "forced_128_fp32dc"),
        # the in-situ diagnostics of a run: ComputeDissipation, the spectrum, divergence norms
        case("diagnostics", (256, 128, 128), "fp64", up, 1, "diagnostics_256x128x128_fp64"),
    ]


# largest grid (log2 of the cells) and steps of the drawn cases of each kind
DRAWN = {"step": (24, 8), "short_run": (20, 50), "run": (24, 12), "sphere": (22, 12), "moving": (21, 8),
         "rollout_grad": (21, 16), "obstacle_grad": (22, 4), "poisson": (24, 1), "forced": (21, 6),
         "diagnostics": (23, 1)}


def draw(rng):
    """One more case: any kind, precision and scheme, every accepted grid (powers
    of two, so spread over their logarithm, mostly not cubes)."""
    while True:
        kind = rng.choice(sorted(DRAWN))
        top, steps = DRAWN[kind]
        e = [rng.randint(4, 8) for _ in range(3)]
        if kind in SPHERE_KINDS:  # x is the long side, the others at least half of it: the box holds the sphere
            e[0] = rng.randint(6, 8)
            e[1:] = [e[0] - rng.randint(0, 1) for _ in range(2)]
        if not 12 <= sum(e) <= top:
            continue
        precision = rng.choice(["fp64", "fp32_dc"])
        if precision == "fp32_dc" and e[0] < 5:
            continue
        scheme = rng.choice(["upwind3_rk2", "upwind3_rk2", "ref"])
        n = rng.randint(max(1, steps // 2), steps)
        return case(kind, tuple(1 << k for k in e), precision, scheme, n)


# ---- inputs --------------------------------------------------------------------
def extent(c):
    return 2.0 if c["kind"] in SPHERE_KINDS else 2 * math.pi


def spacing(c):
    return extent(c) / max(c["nx"], c["ny"], c["nz"])


def viscosity(c):
    nu = {"short_run": 0.01, "step": 5e-3, "rollout_grad": 5e-3, "sphere": 2 * RADIUS / 300,
          "moving": 2 * RADIUS / 300, "obstacle_grad": 2 * RADIUS / 300}.get(c["kind"], 1e-3)
    # central differences with explicit Euler are stable for nu >= u^2 dt / 2
    return max(nu, 0.25 * spacing(c)) if c["scheme"] == "ref" else nu


def cfl(c):
    return 0.5 if c["kind"] == "short_run" and c["scheme"] != "ref" else 0.1


def centres(c):
    h = spacing(c)
    ax = [(torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * h for n in (c["nz"], c["ny"], c["nx"])]
    return torch.meshgrid(*ax, indexing="ij")


def solenoidal(c, seed, k0, rms):
    """Random phases, E(k) ~ k^4 exp(-2 (k/k0)^2) in grid wavenumbers of the longest
    side, free of the central-difference divergence, (3, nz, ny, nx) FP64."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = (c["nz"], c["ny"], c["nx"])
    big = max(n)
    idx = [torch.fft.fftfreq(n[0], 1.0 / n[0], device=DEV, dtype=torch.float64)[:, None, None],
           torch.fft.fftfreq(n[1], 1.0 / n[1], device=DEV, dtype=torch.float64)[None, :, None],
           torch.fft.rfftfreq(n[2], 1.0 / n[2], device=DEV, dtype=torch.float64)[None, None, :]]
    k2 = sum((i * (big / m)) ** 2 for i, m in zip(idx, n))
    amp = torch.sqrt(k2 * torch.exp(-2.0 * k2 / k0 ** 2))  # sqrt(E / k^2)
    white = torch.randn((3,) + n, generator=g, device=DEV, dtype=torch.float64)
    F = [torch.fft.rfftn(white[q]) * amp for q in range(3)]
    s = [torch.sin(2 * math.pi * i / m) + 0 * k2 for i, m in zip(idx, n)][::-1]  # x, y, z
    s2 = s[0] ** 2 + s[1] ** 2 + s[2] ** 2
    dot = sum(a * b for a, b in zip(s, F)) / torch.where(s2 == 0, 1.0, s2)
    u = torch.stack([torch.fft.irfftn(f - a * dot, s=n) for f, a in zip(F, s)])
    return u * (rms / torch.sqrt((u * u).mean()))


def taylor_green(c):
    X, Y, Z = (a * (max(c["nx"], c["ny"], c["nz"]) / m)  # one period along every side
               for a, m in zip(centres(c)[::-1], (c["nx"], c["ny"], c["nz"])))
    return torch.stack([torch.sin(X) * torch.cos(Y) * torch.cos(Z), -torch.cos(X) * torch.sin(Y) * torch.cos(Z),
                        torch.zeros_like(X)])


def initial(c, seed):
    """The initial velocity, rounded to the storage type, as FP64."""
    kind = c["kind"]
    if kind in SPHERE_KINDS:  # (nearly) at rest in the lab frame: the sphere starts the flow
        u = solenoidal(c, seed, 8.0, 0.05)
    elif kind in ("short_run", "rollout_grad"):
        u = taylor_green(c) + solenoidal(c, seed, 4.0, 0.05)
    else:
        u = solenoidal(c, seed, 4.0, 1.0)
    return u.float().double() if c["precision"] == "fp32_dc" else u


def fixed_dts(c):
    """The fixed time steps of the differentiable rollouts."""
    return [0.1 * spacing(c) / (1.2 if c["kind"] == "rollout_grad" else 1.5)] * c["steps"]


def make_sim(c):
    sd = cup.SimulationData(CFL=cfl(c), cells=(c["nx"], c["ny"], c["nz"]))
    sd.extent, sd.nu, sd.rampup, sd.DLM, sd.lambda_ = extent(c), viscosity(c), 0, 0.0, 1.0
    sd.scheme, sd.precision = c["scheme"], c["precision"]
    if c["kind"] in SPHERE_KINDS:
        sd.lambda_, sd.bImplicitPenalization = 1e6, True
    if c["kind"] == "forced":
        sd.turbKinEn_target = 1.6  # a little above the 3/2 of u_rms = 1
    sim = cup.Simulation(sd)
    if c["kind"] in SPHERE_KINDS:
        fixed = c["kind"] != "moving"
        sim.add_obstacle(cup.Sphere(radius=RADIUS, position=CENTRE, enforcedVelocity=(1.0, 0.0, 0.0),
                                    bForcedInSimFrame=(True, True, True), bFixFrameOfRef=(fixed, fixed, fixed)))
    sim.bind_torch_stream()
    return sim


def prepare(c, seed):
    u = initial(c, seed)
    sim = make_sim(c)
    s = {"case": dict(c), "sim": sim}
    raw = u.to(sim.storage_dtype)
    if c["kind"] == "poisson":
        s["rhs"] = poisson_rhs(c, seed)
        return s
    if c["kind"] in ("short_run", "moving"):
        s["u0"] = raw
        return s
    if c["kind"] == "rollout_grad":
        s["u0"] = raw.requires_grad_(True)
        s["target"] = initial(c, seed + 7919).to(sim.storage_dtype)
        return s
    sim.set_velocity(u[0], u[1], u[2])
    sim.run_steps(SPIN_UP[c["kind"]])
    if c["kind"] == "obstacle_grad":  # the drag over a window of the developing flow
        s["u0"] = sim.velocity_raw()
    return s


def poisson_rhs(c, seed):
    """h^3 times a smooth source with white noise on top, zero mean."""
    u = solenoidal(c, seed, 6.0, 1.0)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    f = u[0] * u[1] + 0.01 * torch.randn(u[0].shape, generator=g, device=DEV, dtype=torch.float64)
    return (f - f.mean()) * spacing(c) ** 3


# ---- one pass --------------------------------------------------------------------
def run(s):
    c, sim = s["case"], s["sim"]
    kind = c["kind"]
    if kind == "poisson":
        p = torch.empty_like(s["rhs"])
        sim.bind_torch_stream()
        L.check(L.lib().cup_poisson_solve_field(sim._h, ctypes.c_void_p(s["rhs"].data_ptr()),
                                                ctypes.c_void_p(p.data_ptr()), L.CUP_WHERE_DEVICE), sim._h, "poisson")
        # with FP32 correction solves the solution is good to their tolerance
        return {"p": p if c["precision"] == "fp64" else p.float()}
    if kind == "step":
        for _ in range(c["steps"]):
            st = sim.timestep(sim.calcMaxTimestep())
        return {"u": sim.velocity_raw(), "umax": st.umax, "ke": st.kinetic_energy}
    if kind in ("run", "forced"):
        st = sim.run_steps(c["steps"])
        return {"u": sim.velocity_raw(), "umax": st.umax, "ke": st.kinetic_energy}
    if kind == "sphere":
        st = sim.run_steps(c["steps"])
        return {"u": sim.velocity_raw(), "umax": st.umax, "drag": float(st.force[0])}
    if kind == "short_run":
        sim.set_velocity_raw(s["u0"])
        st = sim.run_steps(c["steps"])
        return {"u": sim.velocity_raw(), "umax": st.umax, "ke": st.kinetic_energy}
    if kind == "moving":
        L.check(L.lib().cup_set_sphere_position(sim._h, (ctypes.c_double * 3)(*CENTRE)), sim._h, "position")
        sim.set_velocity_raw(s["u0"])
        for _ in range(c["steps"]):
            dt = sim.calcMaxTimestep()
            for op in sim.pipeline[:6]:  # CreateObstacles ... Penalization
                op(dt)
        return {"u": sim.velocity_raw(), "drag": float(sim.pipeline[5].force_torque[0])}
    if kind == "rollout_grad":
        s["u0"].grad = None
        uT = adjoint.rollout(sim, s["u0"], fixed_dts(c), checkpoint_every=8)
        (0.5 * (uT - s["target"]).square().sum()).backward()
        return {"u": uT.detach(), "grad": s["u0"].grad}
    if kind == "obstacle_grad":
        n = c["steps"]
        g_u, g_chi, g_vel, forces = adjoint.obstacle_gradients(sim, s["u0"], fixed_dts(c), (1.0 / n, 0.0, 0.0))
        t = sim.storage_dtype
        return {"g_u": g_u, "g_chi": g_chi.to(t), "g_vel": g_vel.to(t), "drag": [float(f[0]) for f in forces]}
    if kind == "diagnostics":
        spec = sim.spectral_analysis()
        d = sim.diagnostics()
        t = np.float64 if c["precision"] == "fp64" else np.float32
        return {"dissipation": np.array(list(sim.compute_dissipation().values()), dtype=t),
                "spectrum": spec["spectrum"].astype(t),
                "stats": np.array([spec[k] for k in ("tke", "eps", "uprime", "lambda", "Re_lambda", "l_integral",
                                                     "tau_integral")], dtype=t),
                "norms": np.array([d["ke"], d["div_l2"], d["div_max"]], dtype=t)}
    raise ValueError(kind)


def work(c):
    """Per step: the velocity read and written and the pressure written, and the
    operations of the advection stages and of the Poisson solve's transforms."""
    n = c["nx"] * c["ny"] * c["nz"]
    w = 4 if c["precision"] == "fp32_dc" else 8
    stages = 2 if c["scheme"] == "upwind3_rk2" else 1
    fft = 2 * 2.5 * math.log2(n)
    step_b, step_f = (6 * w + 8) * n, (stages * 110 + fft + 20) * n
    kind, k = c["kind"], c["steps"]
    if kind == "poisson":
        return {"bytes": 16 * n, "flops": fft * n}
    if kind == "diagnostics":
        return {"bytes": (3 * w + 8) * n, "flops": (1.5 * fft + 150) * n}
    if kind == "rollout_grad":  # forward, and per backward step its state in, the adjoint in and out
        return {"bytes": k * (step_b + 9 * w * n), "flops": 3 * k * step_f}
    if kind == "obstacle_grad":
        return {"bytes": k * (step_b + 9 * w * n) + 8 * n, "flops": 4 * k * step_f}
    if kind == "forced":
        return {"bytes": k * step_b, "flops": k * (step_f + 3 * fft * n)}
    return {"bytes": k * step_b, "flops": k * step_f}


# ---- the same in plain FP64 torch ---------------------------------------------------
def sh(f, axis, k):
    """f at the cell k further along x (0), y (1) or z (2), periodic."""
    return torch.roll(f, -k, dims=2 - axis)


def advect(u, h, nu, dt, uinf, scheme):
    """u + dt A(u) for all three components."""
    a = [u[q] + uinf[q] for q in range(3)]
    facD = nu / h * (dt / h)
    out = []
    for q in range(3):
        f = u[q]
        adv, lap = 0.0, -6.0 * f
        for d in range(3):
            m1, p1 = sh(f, d, -1), sh(f, d, 1)
            lap = lap + m1 + p1
            if scheme == "ref":
                adv = adv + a[d] * (p1 - m1)
            else:
                m2, p2 = sh(f, d, -2), sh(f, d, 2)
                adv = adv + a[d] * torch.where(a[d] > 0, 2 * p1 + 3 * f - 6 * m1 + m2, -p2 + 6 * p1 - 3 * f - 2 * m1)
        facA = -dt / (2 * h) if scheme == "ref" else -dt / (6 * h)
        out.append(f + facA * adv + facD * lap)
    return torch.stack(out)


def advance(u, h, nu, dt, uinf, scheme):
    u1 = advect(u, h, nu, dt, uinf, scheme)
    return u1 if scheme == "ref" else 0.5 * (u + advect(u1, h, nu, dt, uinf, scheme))


def solve(b, h):
    """p with h/4 (sum over the axes of p(+2) - 2 p + p(-2)) = b off the 8 null modes."""
    nz, ny, nx = b.shape
    cs = [torch.cos(4 * math.pi / m * torch.arange(m, device=DEV, dtype=torch.float64)) for m in (nx, ny, nz)]
    den = 2 * (cs[0][None, None, : nx // 2 + 1] + cs[1][None, :, None] + cs[2][:, None, None]) - 6
    null = torch.zeros_like(den)
    for z in (0, nz // 2):
        for y in (0, ny // 2):
            for x in (0, nx // 2):
                null[z, y, x] = 1.0
    f = torch.where(null > 0, 0.0, 4.0 / h / torch.where(null > 0, 1.0, den))
    return torch.fft.irfftn(torch.fft.rfftn(b) * f, s=b.shape)


def central(f, d):
    return sh(f, d, 1) - sh(f, d, -1)


def sphere_chi(c, pos):
    h = spacing(c)
    Z, Y, X = centres(c)

    def sdf(x, y, z):
        return RADIUS - torch.sqrt((x - pos[0]) ** 2 + (y - pos[1]) ** 2 + (z - pos[2]) ** 2)

    s = sdf(X, Y, Z)
    dU, dI = [], []
    for d in range(3):
        P, M = sh(s, d, 1), sh(s, d, -1)
        dU.append((P - M) * (0.5 / h))
        dI.append((P.clamp(min=0) - M.clamp(min=0)) * (0.5 / h))
    X_ = sum(a * b for a, b in zip(dI, dU)) / (sum(a * a for a in dU) + EPS)
    return torch.where((s > 2 * h) | (s < -2 * h), (s > 0).double(), X_)


def one_step(c, u, dt, uinf=(0.0, 0.0, 0.0), chi=None, vel=None, target=0.0):
    """The step's new velocity, pressure and penalization force."""
    h, lam = spacing(c), 1e6
    u = advance(u, h, viscosity(c), dt, uinf, c["scheme"])
    if target:
        n = u[0].numel()
        tke = 0.5 * (u * u).sum() / n
        wf = [2 * math.pi / (m * h) for m in (c["nz"], c["ny"], c["nx"])]
        k = [torch.fft.fftfreq(c["nz"], 1.0 / c["nz"], device=DEV, dtype=torch.float64)[:, None, None] * wf[0],
             torch.fft.fftfreq(c["ny"], 1.0 / c["ny"], device=DEV, dtype=torch.float64)[None, :, None] * wf[1],
             torch.fft.rfftfreq(c["nx"], 1.0 / c["nx"], device=DEV, dtype=torch.float64)[None, None, :] * wf[2]]
        k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
        band = ((k2 > 0) & (k2 <= 4)).double()
        ub = torch.stack([torch.fft.irfftn(torch.fft.rfftn(u[q]) * band, s=u[q].shape) for q in range(3)])
        tkef = 0.5 * (ub * ub).sum() / n
        if tke < target and tkef > 0:
            u = u + (target - tke) / (2 * tkef) * ub
    b = 0.5 * h * h / dt * sum(central(u[d], d) for d in range(3))
    if chi is not None:
        src = -chi * b
        r = b + src
        surf = sum(central(chi.detach(), d) ** 2 for d in range(3)) > 0
        total = src.sum()
        pos, neg = torch.where(surf & (r > 0), r, 0.0).sum(), -torch.where(surf & (r < 0), r, 0.0).sum()
        corr = total / torch.clamp(pos if total > 0 else neg, min=EPS)
        b = torch.where(surf & (r > 0) & (corr > 0), r - corr * r, torch.where(surf & (r < 0) & (corr < 0), r + corr * r, r))
    p = solve(b, h)
    u = u - 0.5 * dt / h * torch.stack([central(p, d) for d in range(3)])
    force = None
    if chi is not None:
        pf = chi * lam / (1 + lam * dt * chi)
        F = [pf * (vel[q] - u[q]) for q in range(3)]
        u = u + dt * torch.stack(F)
        force = [f.sum() * h ** 3 for f in F]
    return u, p, force


def next_dt(c, u, uinf):
    h = spacing(c)
    umax = max(float((u[q] + uinf[q]).abs().max()) for q in range(3))
    return cfl(c) * min(h * h / viscosity(c), h / (umax + 1e-8)), umax


def sphere_box(c):
    """Mask of the cells around the sphere that take part in the obstacle terms."""
    h = spacing(c)
    masks = []
    for pos, n in zip(CENTRE, (c["nx"], c["ny"], c["nz"])):
        r = RADIUS + 3 * h
        lo, hi = math.floor((pos - r) / h - 0.5) - 1, math.ceil((pos + r) / h - 0.5) + 1
        m = torch.zeros(n, dtype=torch.bool, device=DEV)
        m[torch.arange(lo, hi + 1, device=DEV) % n if hi - lo + 1 < n else slice(None)] = True
        masks.append(m)
    return masks[2][:, None, None] & masks[1][None, :, None] & masks[0][None, None, :]


def exact(c, seed):
    kind = c["kind"]
    if kind == "poisson":
        return {"p": solve(poisson_rhs(c, seed), spacing(c))}
    u = initial(c, seed)
    if kind == "rollout_grad":
        with torch.enable_grad():
            u0 = u.requires_grad_(True)
            x = u0
            for dt in fixed_dts(c):
                x = torch.utils.checkpoint.checkpoint(lambda y, dt=dt: one_step(c, y, dt)[0], x, use_reentrant=False)
            (0.5 * (x - initial(c, seed + 7919)).square().sum()).backward()
        return {"u": x.detach(), "grad": u0.grad}
    if kind == "obstacle_grad":
        for _ in range(SPIN_UP[kind]):
            u = one_step(c, u, next_dt(c, u, (-1.0, 0.0, 0.0))[0], (-1.0, 0.0, 0.0), sphere_chi(c, CENTRE),
                         (1.0, 0.0, 0.0))[0]
        with torch.enable_grad():
            u0 = u.requires_grad_(True)
            chi = sphere_chi(c, CENTRE).requires_grad_(True)
            vel = torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device=DEV, requires_grad=True)

            def one(y, x, v, dt):
                a, _, f = one_step(c, y, dt, (-1.0, 0.0, 0.0), x, v)
                return a, f[0]

            x, drag = u0, []
            for dt in fixed_dts(c):
                x, f = torch.utils.checkpoint.checkpoint(one, x, chi, vel, dt, use_reentrant=False)
                drag.append(f)
            (sum(drag) / c["steps"]).backward()
        return {"g_u": u0.grad, "g_chi": torch.where(sphere_box(c), chi.grad, 0.0), "g_vel": vel.grad,
                "drag": [float(f) for f in drag]}
    chi = vel = None
    uinf, pos = (0.0, 0.0, 0.0), list(CENTRE)
    if kind in SPHERE_KINDS:
        vel, chi = (1.0, 0.0, 0.0), sphere_chi(c, pos)
        uinf = (0.0, 0.0, 0.0) if kind == "moving" else (-1.0, 0.0, 0.0)
    target = 1.6 if kind == "forced" else 0.0
    steps = SPIN_UP.get(kind, 0) + (0 if kind == "diagnostics" else c["steps"])
    p = force = None
    for _ in range(steps):
        dt, _ = next_dt(c, u, uinf)
        if kind == "moving":
            pos[0] += dt * vel[0]
            chi = sphere_chi(c, pos)
        u, p, force = one_step(c, u, dt, uinf, chi, vel, target)
    if kind == "diagnostics":
        return exact_diagnostics(c, u, p)
    out = {"u": u}
    if kind != "moving":
        out["umax"] = next_dt(c, u, uinf)[1]
    if chi is None:
        out["ke"] = float(0.5 * (u * u).sum() * spacing(c) ** 3)
    else:
        out["drag"] = float(force[0])
    return out


def exact_diagnostics(c, u, p):
    h, nu = spacing(c), viscosity(c)
    n, h3 = p.numel(), h ** 3
    Z, Y, X = centres(c)
    P = [X - c["nx"] * h / 2, Y - c["ny"] * h / 2, Z - c["nz"] * h / 2]
    D = [[central(u[q], d) / (2 * h) for d in range(3)] for q in range(3)]  # D[q][d] = d u_q / d x_d
    W = [D[2][1] - D[1][2], D[0][2] - D[2][0], D[1][0] - D[0][1]]
    cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]  # noqa: E731
    pp, pw = sum(a * a for a in P), sum(a * b for a, b in zip(P, W))
    lap = [sum(sh(u[q], d, 1) + sh(u[q], d, -1) for d in range(3)) / h ** 2 - 6 * u[q] / h ** 2 for q in range(3)]
    S2 = sum((0.5 * (D[q][d] + D[d][q])) ** 2 for q in range(3) for d in range(3))
    uu = sum(u[q] * u[q] for q in range(3))
    R = [h3 * w.sum() for w in W]
    R += [h3 / 2 * a.sum() for a in cross(P, W)]
    R += [h3 * u[q].sum() for q in range(3)]
    R += [h3 / 3 * (P[q] * pw - W[q] * pp).sum() for q in range(3)]
    R += [h3 * a.sum() for a in cross(P, u)]
    R += [-h3 * sum(central(p, d) / (2 * h) * u[d] for d in range(3)).sum(),
          h3 * nu * (sum(a * u[q] for q, a in enumerate(lap)) + 2 * S2).sum(),
          h3 * sum(W[q] * u[q] for q in range(3)).sum(), h3 * uu.sum() / 2, torch.sqrt(sum(w * w for w in W)).sum()]
    # shell spectrum over all modes of the full complex transform
    E = sum(torch.fft.fftn(u[q]).abs() ** 2 for q in range(3)) * 0.5 / n ** 2
    i = [torch.fft.fftfreq(m, 1.0 / m, device=DEV, dtype=torch.float64) for m in (c["nz"], c["ny"], c["nx"])]
    kind2 = i[0][:, None, None] ** 2 + i[1][None, :, None] ** 2 + i[2][None, None, :] ** 2
    wf = [2 * math.pi / (m * h) for m in (c["nz"], c["ny"], c["nx"])]
    k2 = (i[0][:, None, None] * wf[0]) ** 2 + (i[1][None, :, None] * wf[1]) ** 2 + (i[2][None, None, :] * wf[2]) ** 2
    nyq = max(c["nx"], c["ny"], c["nz"]) // 2
    b = torch.floor(torch.sqrt(kind2) * ((nyq - 1) / nyq)).long()
    ok = (kind2 < nyq ** 2) & (b < nyq - 1)
    spectrum = torch.zeros(nyq - 1, dtype=torch.float64, device=DEV).index_add_(0, b[ok], E[ok])
    tke = float(E.sum())
    eps = nu * float(sum(w * w for w in W).sum()) / n
    up = math.sqrt(2 * tke / 3)
    lam = math.sqrt(15 * nu / eps) * up
    li = float(torch.where(k2 > 0, E / torch.sqrt(torch.where(k2 > 0, k2, 1.0)), 0.0).sum()) / tke
    div = sum(D[d][d] for d in range(3))
    return {"dissipation": torch.stack(R), "spectrum": spectrum,
            "stats": torch.tensor([tke, eps, up, lam, up * lam / nu, li, li / up], dtype=torch.float64),
            "norms": torch.tensor([float(0.5 * uu.sum() * h3), math.sqrt(float((div * div).sum()) * h3),
                                   float(div.abs().max())], dtype=torch.float64)}
