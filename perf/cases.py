"""Performance cases: what a program does with this framework, as measurable passes.

A case is a dict of plain values.  `prepare` makes, from a seed alone, what a
program holds before the call (initial conditions on the GPU, a context under
way, a cooling table); `run` is one pass through the public entry points and
returns its results; `work` counts the bytes and operations the pass cannot do
without; `exact` gives the results in 64 bits with plain torch where they have
such a value.

Results of the mixed-precision path are handed over as float32 (its pair sums
are FP32, and the snapshot files hold float32), except the positions, which it
keeps in FP64; results of the FP64 path and of the drop-in functions as float64.

Kinds:
  step      the time loop on the GPU: `steps` KDK steps of one Evrard sphere,
            then the state read out (the serial driver's loop)
  kh        the same for the periodic Kelvin-Helmholtz slab (hydro only,
            Balsara switch, the MPI driver's order)
  ensemble  one step of a batch of independent Evrard clouds of uneven sizes
  host      one step with the state in page-locked host arrays, moved in and
            out by the call (the reference loop's NumPy arrays)
  start     the start of a run: particles loaded, sorted, tree built, h found
            from nothing, all forces (set_particles + first_step)
  forces    forces for an integrator of the caller's own: new positions and
            velocities in, density, hydro and gravity with potential out, at
            the caller's h
  dropin    one iteration of the reference's CPU driver through the drop-in
            SPH functions (h, density, acceleration, du/dt; FP64)
  gravsum   the drop-in's gravity, the FP64 direct sum in the reference's order
  cooling   the heating/cooling step on the production driver's float arrays
"""
import math

import numpy as np
import torch

from sph_3_b200 import Config, Context, cooling, libsx

DEV = "cuda"
GAMMA = 5.0 / 3.0
DT = 1e-4
NGB = 64
COOL_DIMS = (12, 60, 40, 3, 12, 16)  # N_kpc, N_T, N_nH, N_Z, N_M, N_t
UNITS = dict(unit_density_cgs=1e-24, unit_time_s=3e13, unit_u_cgs=1e12, unit_length_cm=3.086e21)

_stream = None


def _side_stream():
    """The stream every context of the program works on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a small test sphere (the sizes of the reference's quick runs): 8
        # steps between outputs, where launches and latency count
        {"name": "step_2k", "kind": "step", "n": 2000, "precision": "mixed", "visc": "signal", "steps": 8},
        # an ordinary run of a ragged size
        {"name": "step_50k", "kind": "step", "n": 50021, "precision": "mixed", "visc": "balsara", "steps": 2},
        # the headline: Evrard collapse of a million particles
        {"name": "step_1m", "kind": "step", "n": 1048576, "precision": "mixed", "visc": "signal", "steps": 1},
        # the plain FP64 path the mixed one is compared with
        {"name": "step_fp64", "kind": "step", "n": 131072, "precision": "fp64", "visc": "signal", "steps": 1},
        # the periodic slab at its full size, the largest single system
        {"name": "kh_4m", "kind": "kh", "n": 4194304, "precision": "mixed"},
        # a batch of clouds, sizes log-uniform in [2048, 65536]
        {"name": "ensemble_64", "kind": "ensemble", "clouds": 64, "n_min": 2048, "n_max": 65536},
        # the state in host arrays, FP64 as the reference's loop keeps it
        {"name": "host_100k", "kind": "host", "n": 100000, "precision": "fp64"},
        # the start of a run
        {"name": "start_250k", "kind": "start", "n": 250007, "precision": "mixed"},
        # forces for the caller's own integrator
        {"name": "forces_100k", "kind": "forces", "n": 100003, "precision": "mixed", "visc": "signal"},
        # the reference's CPU configuration (N = 10,000) through the drop-in
        {"name": "dropin_10k", "kind": "dropin", "n": 10000},
        {"name": "gravsum_10k", "kind": "gravsum", "n": 10000},
        # the production driver's heating/cooling on a large run's gas
        {"name": "cooling_2m", "kind": "cooling", "n": 2000003},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "kh", "ensemble", "host", "start", "forces", "dropin", "gravsum",
                       "cooling"])
    if kind == "step":
        prec = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        n = _logint(rng, 1000, 1000000 if prec == "mixed" else 200000)
        return {"kind": kind, "n": n, "precision": prec, "visc": rng.choice(["signal", "mg83", "balsara"]),
                "steps": 8 if n < 8000 else (2 if n < 100000 else 1)}
    if kind == "kh":
        return {"kind": kind, "n": _logint(rng, 60000, 3000000), "precision": "mixed"}
    if kind == "ensemble":
        return {"kind": kind, "clouds": rng.randint(3, 64), "n_min": 2048, "n_max": rng.randint(8192, 65536)}
    if kind == "host":
        return {"kind": kind, "n": _logint(rng, 5000, 150000), "precision": "fp64"}
    if kind == "start":
        return {"kind": kind, "n": _logint(rng, 3000, 400000), "precision": rng.choice(["mixed", "fp64"])}
    if kind == "forces":
        return {"kind": kind, "n": _logint(rng, 3000, 200000), "precision": "mixed",
                "visc": rng.choice(["signal", "mg83"])}
    if kind == "dropin":
        return {"kind": kind, "n": _logint(rng, 600, 20000)}
    if kind == "gravsum":
        return {"kind": kind, "n": _logint(rng, 600, 30000)}
    return {"kind": kind, "n": _logint(rng, 50000, 3000000)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _evrard(n, seed, M=1.0, R=1.0):
    """An Evrard sphere (rho ~ 1/r) falling in, with a little turbulence and a
    spread of internal energies, as a run meets it under way."""
    g = _gen(seed)
    f64 = dict(dtype=torch.float64, device=DEV, generator=g)
    r = R * torch.sqrt(torch.rand(n, **f64))
    d = torch.randn(n, 3, **f64)
    d /= torch.linalg.norm(d, dim=1, keepdim=True)
    pos = d * r[:, None]
    vel = -0.4 * pos / R + 0.05 * torch.randn(n, 3, **f64)
    u = 0.05 * (M / R) * (0.7 + 0.6 * torch.rand(n, **f64))
    m = torch.full((n,), M / n, dtype=torch.float64, device=DEV)
    return dict(pos=pos.contiguous(), vel=vel.contiguous(), m=m, u=u)


def _evrard_h(pos, n):
    """h from the profile's number density n(r) = N / (2 pi r)."""
    r = torch.linalg.norm(pos, dim=1).clamp_min(0.3 / math.sqrt(n) + 0.01)
    return 0.5 * (3.0 * NGB * 2.0 * math.pi * r / (4.0 * math.pi * n)) ** (1.0 / 3.0)


def _kh(n, seed):
    """The Kelvin-Helmholtz slab [0,1] x [0,1] x [0,1/16]: density 2 inside
    |y - 0.5| < 0.25, 1 outside, sheared, on lattices jittered by a tenth of
    their spacing (the state a few sound crossings in)."""
    g = _gen(seed)
    f64 = dict(dtype=torch.float64, device=DEV)
    Lz = 1.0 / 16.0
    m = 1.5 * Lz / n
    parts = []
    for rho, ylo, yhi in ((2.0, 0.25, 0.75), (1.0, 0.0, 0.25), (1.0, 0.75, 1.0)):
        d = (m / rho) ** (1.0 / 3.0)
        nx, ny, nz = math.ceil(1.0 / d), math.ceil((yhi - ylo) / d), math.ceil(Lz / d)
        gx = (torch.arange(nx, **f64) + 0.5) / nx
        gy = ylo + (torch.arange(ny, **f64) + 0.5) * ((yhi - ylo) / ny)
        gz = (torch.arange(nz, **f64) + 0.5) * (Lz / nz)
        p = torch.stack(torch.meshgrid(gx, gy, gz, indexing="ij"), dim=-1).reshape(-1, 3)
        parts.append(p + 0.1 * d * torch.randn(p.shape, generator=g, **f64))
    pos = torch.cat(parts)
    keep = torch.randperm(pos.shape[0], device=DEV, generator=g)[:n].sort().values
    pos = pos[keep]
    box = torch.tensor([1.0, 1.0, Lz], **f64)
    pos = (pos - torch.floor(pos / box) * box).contiguous()
    pos = torch.where(pos >= box, torch.zeros_like(pos), pos)
    n = pos.shape[0]
    inner = (pos[:, 1] - 0.5).abs() < 0.25
    vel = torch.zeros(n, 3, **f64)
    vel[:, 0] = torch.where(inner, 0.5, -0.5)
    vel[:, 1] = 0.01 * torch.sin(4.0 * math.pi * pos[:, 0])
    u = 2.5 / ((GAMMA - 1.0) * torch.where(inner, 2.0, 1.0).to(torch.float64))
    return dict(pos=pos, vel=vel, m=torch.full((n,), m, **f64), u=u, box=(1.0, 1.0, Lz))


def _cloud_sizes(case):
    """Sizes log-uniform in [n_min, n_max], spread evenly over the clouds."""
    k = case["clouds"]
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [int(math.exp(lo + (hi - lo) * ((i * 0.6180339887498949) % 1.0))) for i in range(k)]


# ------------------------------------------------------------------ prepare
def _under_way(ctx, ic, warm):
    """A context with the particles loaded, the first step done and the loop
    running (its step captured)."""
    s = _side_stream()
    torch.cuda.synchronize()  # the initial conditions are ready
    with torch.cuda.stream(s):
        ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"])
        ctx.first_step(DT)
        if warm:
            ctx.step(DT, 3, stream=s.cuda_stream)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "step":
        ctx = Context(Config(precision=case["precision"], visc=case["visc"]))
        st["ctx"] = _under_way(ctx, _evrard(case["n"], seed), True)
    elif kind == "kh":
        ic = _kh(case["n"], seed)
        ctx = Context(Config(precision=case["precision"], visc="balsara", step_order="mpi4", gravity=False,
                             box=ic["box"]))
        st["ctx"] = _under_way(ctx, ic, True)
    elif kind == "ensemble":
        sizes = _cloud_sizes(case)
        rng = np.random.default_rng(seed)
        ics = [_evrard(k, seed * 1009 + i, M=float(rng.uniform(0.5, 2.0)), R=float(rng.uniform(0.5, 2.0)))
               for i, k in enumerate(sizes)]
        ic = {f: torch.cat([c[f] for c in ics]).contiguous() for f in ("pos", "vel", "m", "u")}
        ctx = Context(Config(precision="mixed", walk_warps=2))
        ctx.set_clouds(sizes)
        st["ctx"] = _under_way(ctx, ic, True)
    elif kind == "host":
        ctx = Context(Config(precision=case["precision"]))
        _under_way(ctx, _evrard(case["n"], seed), False)
        arrays = {}
        for f in ("pos", "vel", "u", "h", "acc", "dudt_prev"):
            v = ctx.get_field(f)
            arrays[f] = torch.empty(v.shape, dtype=torch.float64, pin_memory=True)
            arrays[f].copy_(torch.from_numpy(v))
        st.update(ctx=ctx, arrays=arrays)
        for _ in range(4):  # the loop is running
            ctx.step_io(DT, arrays, arrays)
    elif kind == "start":
        st.update(ctx=Context(Config(precision=case["precision"])), ic=_evrard(case["n"], seed))
    elif kind == "forces":
        ic = _evrard(case["n"], seed)
        ctx = Context(Config(precision=case["precision"], visc=case["visc"]))
        ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"], h=_evrard_h(ic["pos"], case["n"]))
        st.update(ctx=ctx, ic=ic)
    elif kind in ("dropin", "gravsum"):
        ic = _evrard(case["n"], seed)
        g = _gen(seed + 7)
        st["ic"] = ic
        # the previous step's h, a few 0.3 % steps away
        st["h"] = _dropin_h(ic["pos"]) * (0.97 + 0.06 * torch.rand(case["n"], dtype=torch.float64, device=DEV,
                                                                   generator=g))
        st["eps"] = torch.full((case["n"],), 0.01, dtype=torch.float64, device=DEV)
    elif kind == "cooling":
        st.update(_cooling_state(case, seed))
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return st


def _dropin_h(pos):
    """Half the radius that holds 50 particles, from the nearest neighbours."""
    n = pos.shape[0]
    h = torch.empty(n, dtype=torch.float64, device=DEV)
    for b in range(0, n, 4096):
        d = torch.cdist(pos[b:b + 4096], pos, compute_mode="donot_use_mm_for_euclid_dist")
        h[b:b + 4096] = 0.5 * d.kthvalue(min(51, n), dim=1).values
    return h


def _cooling_state(case, seed):
    n = case["n"]
    g = _gen(seed)
    f32 = dict(dtype=torch.float32, device=DEV, generator=g)
    return dict(raw=cooling.seeded_table(seed=seed, dims=COOL_DIMS) if case.get("raw") else None,
                table=None if case.get("raw") else cooling.CoolTable(cooling.seeded_table(seed=seed, dims=COOL_DIMS)),
                xyz=tuple(torch.rand(n, **f32) * 4 - 2 for _ in range(3)),
                rho=10.0 ** (torch.rand(n, **f32) * 8 - 4), u0=10.0 ** (torch.rand(n, **f32) * 6 - 3),
                u=torch.empty(n, dtype=torch.float32, device=DEV),
                typ=torch.zeros(n, dtype=torch.int32, device=DEV))


# ------------------------------------------------------------------ run
def _read(ctx, fields, mixed):
    out = {}
    for f in fields:
        v = ctx.get_field(f, device=True)
        out[f] = v.float() if mixed and f != "pos" else v
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "kh", "ensemble"):
        s = _side_stream()
        ctx = state["ctx"]
        with torch.cuda.stream(s):
            ctx.step(DT, case.get("steps", 1), stream=s.cuda_stream)
            return _read(ctx, ("pos", "vel", "u", "h", "rho", "acc"), ctx.config.precision == "mixed")
    if kind == "host":
        state["ctx"].step_io(DT, state["arrays"], state["arrays"])
        return state["arrays"]
    if kind == "start":
        s = _side_stream()
        ctx, ic = state["ctx"], state["ic"]
        with torch.cuda.stream(s):
            ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"])
            ctx.first_step(DT)
            return _read(ctx, ("h", "nngb", "rho", "acc_g", "phi", "acc_sph", "dudt", "u"),
                         ctx.config.precision == "mixed")
    if kind == "forces":
        s = _side_stream()
        ctx, ic = state["ctx"], state["ic"]
        with torch.cuda.stream(s):
            ctx.set_field("pos", ic["pos"])
            ctx.set_field("vel", ic["vel"])
            ctx.compute("density", "gravity", "acc_sph", "dudt")
            return _read(ctx, ("rho", "P", "c", "acc_sph", "dudt", "acc_g", "phi"),
                         ctx.config.precision == "mixed")
    if kind == "dropin":
        ic = state["ic"]
        h = libsx.h_smooth_fast(ic["pos"], state["h"])
        rho = libsx.getDensity(ic["pos"], ic["m"], h)
        P = libsx.getPressure(rho, ic["u"], GAMMA)
        c = torch.sqrt(GAMMA * (GAMMA - 1.0) * ic["u"])
        acc = libsx.getAcc_sph(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], GAMMA, 0.1, 1.0, 2.0)
        dudt = libsx.get_dU(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], GAMMA, 0.1, 1.0, 2.0)
        return dict(h=h, rho=rho, P=P, acc=acc, dudt=dudt)
    if kind == "gravsum":
        ic = state["ic"]
        return libsx.getAcc_g_smth(ic["pos"], ic["m"], 1.0, state["eps"])
    state["u"].copy_(state["u0"])  # the energies the u update left
    return list(cooling.hcooling(state["table"], cooling.Units(**UNITS), DT, state["u"], state["rho"], state["xyz"],
                                 typ=state["typ"]))


# ------------------------------------------------------------------ work
def _step_work(n, precision, gravity, clouds_n=None):
    """Per particle: the state read and written once (FP64: positions,
    velocities, u, its history, du/dt, h, acceleration, masses, softening),
    the key sort's keys and the results; candidate tests and pair terms of
    NGB-neighbour supports, and for gravity the interactions a theta = 0.5
    walk needs (about 55 nodes and particles per level of the tree)."""
    size = clouds_n or n
    flops = n * (8 * NGB * 2 + 20 * NGB + 75 * NGB)
    if gravity:
        flops += n * 40.0 * 55.0 * max(1.0, math.log2(max(size, 8) / 8.0) / 3.0)
    return {"bytes": n * (15 * 8 * 2 + 12 + 6 * 8), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("step", "kh"):
        w = _step_work(case["n"], case["precision"], kind == "step")
        k = case.get("steps", 1)
        return {"bytes": w["bytes"] * k, "flops": w["flops"] * k}
    if kind == "ensemble":
        parts = [_step_work(k, "mixed", True) for k in _cloud_sizes(case)]
        return {f: sum(p[f] for p in parts) for f in ("bytes", "flops")}
    n = case["n"]
    if kind == "host":
        w = _step_work(n, case["precision"], True)
        return {"bytes": w["bytes"] + 2 * 12 * 8 * n, "flops": w["flops"]}
    if kind == "start":
        w = _step_work(n, case["precision"], True)
        return {"bytes": w["bytes"], "flops": w["flops"] + n * 8 * NGB * 3}
    if kind == "forces":
        return _step_work(n, case["precision"], True)
    if kind == "dropin":
        # each of the four functions reads its inputs and writes its result
        return {"bytes": n * 8 * (4 + 1 + 5 + 1 + 11 + 3 + 11 + 1), "flops": n * 50 * (8 * 4 + 20 + 75 + 60)}
    if kind == "gravsum":
        return {"bytes": n * 8 * 8, "flops": 30.0 * n * n}
    nm = COOL_DIMS[4]
    return {"bytes": n * (4 * 6 + 4 + 4 * nm), "flops": n * 60}


# ------------------------------------------------------------------ 64 bits
def _rows(n, most=1 << 26):
    step = max(1, most // n)
    for b in range(0, n, step):
        yield b, min(n, b + step)


def _gravity64(pos, m, eps, want_phi):
    n = pos.shape[0]
    acc = torch.empty(n, 3, dtype=torch.float64, device=DEV)
    phi = torch.empty(n, dtype=torch.float64, device=DEV)
    x, y, z = pos.t().contiguous()
    for b, e in _rows(n):
        dx, dy, dz = x[None] - x[b:e, None], y[None] - y[b:e, None], z[None] - z[b:e, None]
        r = torch.sqrt(dx * dx + dy * dy + dz * dz)
        self_pair = r == 0
        r = torch.where(self_pair, torch.ones_like(r), r)
        q = r / eps
        q2 = q * q
        q3 = q2 * q
        inner = q <= 1.0
        far = q > 2.0
        i3 = 1.0 / (r * r * r)
        fk = torch.where(inner, (4.0 / 3.0 - 1.2 * q2 + 0.5 * q3) / eps ** 3,
                         i3 * (-1.0 / 15.0 + 8.0 / 3.0 * q3 - 3.0 * q2 * q2 + 1.2 * q2 * q3 - q3 * q3 / 6.0))
        fk = torch.where(far, i3, fk) * m[None]
        fk = torch.where(self_pair, torch.zeros_like(fk), fk)
        acc[b:e, 0], acc[b:e, 1], acc[b:e, 2] = (fk * dx).sum(1), (fk * dy).sum(1), (fk * dz).sum(1)
        if want_phi:
            pk = torch.where(inner, -2.0 / eps * (q2 / 3.0 - 0.15 * q2 * q2 + 0.05 * q2 * q3) + 1.4 / eps,
                             -1.0 / (15.0 * r) - (4.0 / 3.0 * q2 - q3 + 0.3 * q2 * q2 - q2 * q3 / 30.0) / eps
                             + 1.6 / eps)
            pk = torch.where(far, 1.0 / r, pk) * m[None]
            phi[b:e] = -torch.where(self_pair, torch.zeros_like(pk), pk).sum(1)
    return acc, phi


def _density64(pos, m, h):
    n = pos.shape[0]
    rho = torch.empty(n, dtype=torch.float64, device=DEV)
    for b, e in _rows(n):
        d = torch.sqrt(((pos[b:e, None, 0] - pos[None, :, 0]) ** 2 + (pos[b:e, None, 1] - pos[None, :, 1]) ** 2
                        + (pos[b:e, None, 2] - pos[None, :, 2]) ** 2))
        hij = 0.5 * (h[b:e, None] + h[None])
        q = d / hij
        W = torch.where(q <= 1.0, 1.0 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2.0 - q).clamp_min(0.0) ** 3)
        rho[b:e] = (m[None] * W / (math.pi * hij ** 3)).sum(1)
    return rho


def _hydro64(pos, vel, rho, P, c, h, m, visc, alpha=1.0, beta=2.0, eta=0.1):
    """Hydro acceleration and du/dt over the pairs inside |r| <= h_i + h_j."""
    n = pos.shape[0]
    acc = torch.zeros(n, 3, dtype=torch.float64, device=DEV)
    dudt = torch.zeros(n, dtype=torch.float64, device=DEV)
    pr = P / (rho * rho)
    for b, e in _rows(n):
        d2 = ((pos[b:e, None, 0] - pos[None, :, 0]) ** 2 + (pos[b:e, None, 1] - pos[None, :, 1]) ** 2
              + (pos[b:e, None, 2] - pos[None, :, 2]) ** 2)
        i, j = torch.nonzero(d2 <= (h[b:e, None] + h[None]) ** 2, as_tuple=True)
        i = i + b
        d = pos[i] - pos[j]
        rr = torch.sqrt((d * d).sum(1))
        hij = 0.5 * (h[i] + h[j])
        q = rr / hij
        nW = torch.where(q <= 1.0, -3.0 + 2.25 * q, -0.75 * (2.0 - q).clamp_min(0.0) ** 2 / (q + 1e-20))
        gW = (nW / (math.pi * hij ** 5))[:, None] * d
        v = vel[i] - vel[j]
        vr = (v * d).sum(1)
        rhoij = 0.5 * (rho[i] + rho[j])
        if visc == "mg83":
            mu = hij * vr / (rr * rr + hij * hij * eta * eta)
            PI = (-alpha * 0.5 * (c[i] + c[j]) * mu + beta * mu * mu) / rhoij
        else:
            w = vr / (rr + 1e-5)
            PI = -0.5 * alpha * (c[i] + c[j] - 3.0 * w) * w / rhoij
        PI = torch.where(vr <= 0.0, PI, torch.zeros_like(PI))
        t = -(m[j] * (pr[i] + pr[j] + PI))[:, None] * gW
        acc.index_add_(0, i, t)
        dudt.index_add_(0, i, m[j] * (pr[i] + 0.5 * PI) * (v * gW).sum(1))
    return acc, dudt


def _h_rule64(pos, h, n_ngb=50, tol=5):
    """h moved by 0.3 % per step until N(r < 2h) is within n_ngb +- tol."""
    n = pos.shape[0]
    out = h.clone()
    for b, e in _rows(n, 1 << 25):
        d = torch.sqrt((pos[b:e, None, 0] - pos[None, :, 0]) ** 2 + (pos[b:e, None, 1] - pos[None, :, 1]) ** 2
                       + (pos[b:e, None, 2] - pos[None, :, 2]) ** 2)
        hb = out[b:e].clone()
        for _ in range(3000):
            cnt = (d < 2.0 * hb[:, None]).sum(1)
            over, under = cnt > n_ngb + tol, cnt < n_ngb - tol
            if not bool((over | under).any()):
                break
            hb = torch.where(over, hb - 0.003 * hb, torch.where(under, hb + 0.003 * hb, hb))
        out[b:e] = hb
    return out


def _nearest(grid, x):
    k = torch.searchsorted(grid, x.contiguous(), right=False)
    last = k >= grid.numel()
    k = k.clamp_max(grid.numel() - 1)
    below = (k - 1).clamp_min(0)
    closer = (grid[below] - x).abs() < (grid[k] - x).abs()
    return torch.where(last, torch.full_like(k, grid.numel() - 1), torch.where((k > 0) & closer, below, k))


def _cooling64(case, seed):
    """The float lookups decide the table cell; the interpolation in 64 bits."""
    s = _cooling_state(dict(case, raw=True), seed)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for k, v in s["raw"].items()}
    units = {k: np.float32(v) for k, v in UNITS.items()}
    x, y, z = s["xyz"]
    r = torch.sqrt(x * x + y * y + z * z) * float(units["unit_length_cm"]) / float(np.float32(3.086e21))
    ik = _nearest(t["kpc"], r)
    nh = s["rho"] * float(units["unit_density_cgs"]) * float(np.float32(0.70)) / float(np.float32(1.6726e-24))
    ih = _nearest(t["nH"], nh)
    it = int(_nearest(t["t"], torch.tensor([float(np.float32(DT) * units["unit_time_s"])], dtype=torch.float32,
                                           device=DEV))[0])
    ucgs = s["u0"] * float(units["unit_u_cgs"])
    iz = 1
    cols = t["uArr"][:, :, :, iz].permute(0, 2, 1).contiguous()  # [kpc][nH][T]
    mine = cols[ik, ih]
    nT = cols.shape[2]
    iu = torch.searchsorted(mine, ucgs[:, None], right=False)[:, 0].clamp_max(nT - 1)
    below = (iu - 1).clamp_min(0)
    ev = t["uEvol"][:, :, :, iz, it].permute(0, 2, 1)
    e2, e1 = ev[ik, ih, iu].double(), ev[ik, ih, below].double()
    hi, lo = mine.gather(1, iu[:, None])[:, 0].double(), mine.gather(1, below[:, None])[:, 0].double()
    f = (ucgs.double() - lo) / torch.where(iu > 0, hi - lo, torch.ones_like(hi))
    new = torch.where(iu > 0, f * e2 + (1.0 - f) * e1, e2)
    ion = t["metalz"][:, :, :, iz, :, it][ik, iu, ih]
    return [new / float(units["unit_u_cgs"]), ion.double()]


def exact(case, seed):
    kind = case["kind"]
    if kind == "forces":
        ic = _evrard(case["n"], seed)
        h = _evrard_h(ic["pos"], case["n"])
        rho = _density64(ic["pos"], ic["m"], h)
        P = (GAMMA - 1.0) * rho * ic["u"]
        c = torch.sqrt(GAMMA * (GAMMA - 1.0) * ic["u"])
        acc, dudt = _hydro64(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], case["visc"])
        acc_g, phi = _gravity64(ic["pos"], ic["m"], 0.01, True)
        return dict(rho=rho, P=P, c=c, acc_sph=acc, dudt=dudt, acc_g=acc_g, phi=phi)
    if kind == "dropin":
        st = prepare(case, seed)
        ic = st["ic"]
        h = _h_rule64(ic["pos"], st["h"])
        rho = _density64(ic["pos"], ic["m"], h)
        P = (GAMMA - 1.0) * rho * ic["u"]
        c = torch.sqrt(GAMMA * (GAMMA - 1.0) * ic["u"])
        acc, dudt = _hydro64(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], "signal")
        return dict(h=h, rho=rho, P=P, acc=acc, dudt=dudt)
    if kind == "gravsum":
        ic = _evrard(case["n"], seed)
        return _gravity64(ic["pos"], ic["m"], 0.01, False)[0]
    if kind == "cooling":
        return _cooling64(case, seed)
    # the steps and the start of a run search h to a window of neighbour
    # counts: which h of the window is found has no exact value, and every
    # other result follows from it
    return None
