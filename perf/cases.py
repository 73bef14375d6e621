"""The workloads this framework's speed is measured on, through its public
entry points: 3-D r2r transforms (R2RPlan), time steps of one instance
(Simulation) and of an ensemble (Ensemble).

A transform case copies the field into a work buffer and transforms it there,
as the reference copies every field into `trans_local` before fftw_execute.
A step case advances the instance by the diagnostics cadence of the reference's
loop, reads the diagnostics and downloads psi, which is what a run writes out
and restarts from (the FP64 cases read rho too, the small ones vz).  Its divv
switch is at step 10 instead of 200, so that the divv quotient and the pressure
coupling are on, as they are in nearly all steps of a long run.  The quotient
divides a difference of two densities by dt, so velocities and L1 carry the
round-off of their type a thousandfold: they are outputs where that leaves them
meaningful digits (FP64, the velocity on the small grids).
"""
import math

import numpy as np
import torch

import smaiso_quasi_b200 as q

ELEM = {"fp64": 8, "fp32": 4}
SWITCH = 10   # divv_switch of the step cases


def listed():
    return [
        # the smallest transform: launch latency
        {"name": "r2r_tiny_fp64", "kind": "r2r", "nx": 16, "ny": 16, "nz": 32, "precision": "fp64", "plan": "CT"},
        # one field of the reference's own 64x64x128 box, inverse with a sine axis
        {"name": "r2r_small_fp32", "kind": "r2r", "nx": 64, "ny": 64, "nz": 128, "precision": "fp32", "plan": "iSTz"},
        # lengths with a factor 3, forward with a sine axis
        {"name": "r2r_ragged_fp64", "kind": "r2r", "nx": 96, "ny": 96, "nz": 192, "precision": "fp64", "plan": "STy"},
        # the headline grid, both directions and types
        {"name": "r2r_large_fp32", "kind": "r2r", "nx": 256, "ny": 256, "nz": 256, "precision": "fp32", "plan": "CT"},
        {"name": "r2r_large_fp64", "kind": "r2r", "nx": 256, "ny": 256, "nz": 256, "precision": "fp64", "plan": "iSTx"},
        # the smallest instance: every kernel of the step is launch-bound
        {"name": "step_tiny_fp64", "kind": "step", "variant": "quasi", "nx": 16, "ny": 16, "nz": 32,
         "precision": "fp64", "ranks": 2, "ic": "planar", "steps": 10},
        # the reference's own box as it runs it: 4 MPI ranks, 50 steps between diagnostics
        {"name": "step_small_fp64", "kind": "step", "variant": "quasi", "nx": 64, "ny": 64, "nz": 128,
         "precision": "fp64", "ranks": 4, "ic": "planar", "steps": 50},
        # a middle grid, undulated layers
        {"name": "step_mid_fp32", "kind": "step", "variant": "quasi", "nx": 128, "ny": 128, "nz": 256,
         "precision": "fp32", "ranks": 1, "ic": "undulated", "steps": 50},
        # the stability variant
        {"name": "step_stb_fp32", "kind": "step", "variant": "stb", "nx": 96, "ny": 96, "nz": 192,
         "precision": "fp32", "ranks": 1, "ic": "stb", "steps": 50},
        # the headline: a 256^3 planar interface, both forms
        {"name": "step_large_fp32", "kind": "step", "variant": "quasi", "nx": 256, "ny": 256, "nz": 256,
         "precision": "fp32", "ranks": 1, "ic": "planar", "steps": 50},
        {"name": "step_large_fp64", "kind": "step", "variant": "quasi", "nx": 256, "ny": 256, "nz": 256,
         "precision": "fp64", "ranks": 1, "ic": "planar", "steps": 50},
        # a stability ensemble: members on the three grids of ensemble.GRIDS
        {"name": "ensemble_fp32", "kind": "ensemble", "members": 6, "precision": "fp32", "steps": 50},
    ]


LENGTHS = (16, 32, 64, 96, 128, 192, 256, 512)


def _grid(rng):
    """A grid of the supported lengths, its cell count log-uniform in 2^13 .. 2^24."""
    want = 2.0 ** rng.uniform(13, 24)
    while True:
        g = [rng.choice(LENGTHS) for _ in range(3)]
        cells = g[0] * g[1] * g[2]
        if want / 1.6 <= cells <= min(want * 1.6, 2 ** 24):
            return g


def draw(rng):
    kind = rng.choice(("r2r", "r2r", "r2r", "step", "step", "step", "ensemble"))
    precision = rng.choice(("fp64", "fp32"))
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 6), "precision": precision, "steps": rng.randint(5, 50)}
    nx, ny, nz = _grid(rng)
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision}
    if kind == "r2r":
        return dict(c, plan=rng.choice(sorted(q.quasi.PLAN_KINDS)))
    variant = rng.choice(("quasi", "quasi", "stb"))
    ic = "stb" if variant == "stb" else rng.choice(("planar", "undulated"))
    return dict(c, variant=variant, ranks=rng.choice((1, 1, 2, 4)), ic=ic, steps=rng.randint(5, 50))


# ---------------------------------------------------------------------------
def _config(c):
    return q.default_config(c["variant"], c["nx"], c["ny"], c["nz"], precision=c["precision"],
                            emulate_ranks=c["ranks"], divv_switch=SWITCH)


def _initial(c, cfg, seed):
    return q.initial_condition(cfg, c["ic"], seed=seed)


def _members(c):
    """(grid, q_h, eps_h) of each ensemble member."""
    out = []
    for m in range(c["members"]):
        g = ((64, 64, 128), (96, 96, 192), (128, 128, 256))[m % 3]
        lx = g[0] * 2.0 * math.pi / 8
        out.append((g, 2.0 * math.pi * (1 + m) / lx, 0.1 - 0.01 * m))
    return out


def _member_setup(c, seed):
    cfgs, psis = [], []
    for m, (g, q_h, eps_h) in enumerate(_members(c)):
        cfg = q.default_config("stb", *g, precision=c["precision"], q_pert=q_h)
        cfgs.append(cfg)
        psis.append(q.initial_condition(cfg, "interface", seed=seed + 97 * m, eps_h=eps_h, q_h=q_h))
    return cfgs, psis


def _field_in(c, seed):
    """A real-space or spectral field: unit-variance values."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float64 if c["precision"] == "fp64" else torch.float32
    return torch.randn(c["nx"], c["ny"], c["nz"], generator=gen, device="cuda", dtype=dt)


def prepare(case, seed):
    c = case
    if c["kind"] == "r2r":
        x = _field_in(c, seed)
        plan = q.R2RPlan(c["nx"], c["ny"], c["nz"], c["plan"], precision=c["precision"])
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        return {"case": c, "x": x, "work": torch.empty_like(x), "plan": plan, "stream": stream}
    if c["kind"] == "step":
        cfg = _config(c)
        sim = q.Simulation(cfg)
        sim.set_psi(_initial(c, cfg, seed))
        sim.init()
        return {"case": c, "sim": sim}
    cfgs, psis = _member_setup(c, seed)
    ens = q.Ensemble(cfgs)
    for s, psi in zip(ens.members, psis):
        s.set_psi(psi)
    ens.init()
    return {"case": c, "ens": ens}


def _out(c, field):
    """A downloaded field in the form's own type."""
    return field if c["precision"] == "fp64" else field.astype(np.float32)


def _outputs(c):
    """What a step case returns."""
    keys = ["mass", "energy", "psi"]
    if c["precision"] == "fp64":
        keys.append("L1")
        if c["variant"] == "quasi":
            keys += ["rho", "vz"] if c["nx"] * c["ny"] * c["nz"] <= 2 ** 20 else ["rho"]
    return keys


def run(state):
    c = state["case"]
    if c["kind"] == "r2r":
        st = state["stream"]
        with torch.cuda.stream(st):
            state["work"].copy_(state["x"])
        state["plan"].execute_device(state["work"].data_ptr(), st.cuda_stream)
        return state["work"]
    if c["kind"] == "step":
        sim = state["sim"]
        sim.step(c["steps"])
        l1, mass, energy = sim.diagnostics()
        got = {"L1": l1, "mass": mass, "energy": energy}
        return {k: got[k] if k in got else _out(c, sim.field(k)) for k in _outputs(c)}
    ens = state["ens"]
    ens.step(c["steps"])
    growth = ens.growth_rates()
    return {"growth": _out(c, growth), "psi": [_out(c, s.field("psi")) for s in ens.members]}


# ---------------------------------------------------------------------------
# 24 transforms a quasi step, 13 a quasi-stb step (sh, three stress, p, three
# velocity, N, psi and its three gradients), each reading and writing its field
# once; a transform is 2.5 N log2 N operations per pencil and axis.
def _transform_work(nx, ny, nz, elem):
    n = nx * ny * nz
    return 2.0 * elem * n, 2.5 * n * math.log2(n)


def work(case):
    c = case
    elem = ELEM[c["precision"]]
    if c["kind"] == "r2r":
        b, f = _transform_work(c["nx"], c["ny"], c["nz"], elem)
        return {"bytes": b, "flops": f}
    grids = [(c["nx"], c["ny"], c["nz"])] if c["kind"] == "step" else [g for g, _, _ in _members(c)]
    transforms = 24 if c.get("variant") == "quasi" else 13
    b = f = 0.0
    for g in grids:
        tb, tf = _transform_work(*g, elem)
        b += c["steps"] * transforms * tb
        f += c["steps"] * transforms * tf
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same in 64 bits by plain torch: transforms as dense products with the
# matrices of FFTW's kinds, the step statement by statement.
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _matrix(kind, n):
    """y = M x for REDFT10, REDFT01, RODFT10, RODFT01 (unnormalised).  Angles are
    reduced exactly as integers: every one is a multiple of pi / 2n."""
    dev = _device()
    k = torch.arange(n, device=dev, dtype=torch.int64)[:, None]
    m = torch.arange(n, device=dev, dtype=torch.int64)[None, :]
    units = {0: k * (2 * m + 1), 1: m * (2 * k + 1), 2: (k + 1) * (2 * m + 1), 3: (m + 1) * (2 * k + 1)}[kind]
    ang = (units % (4 * n)).double() * (math.pi / (2 * n))
    out = 2.0 * (torch.cos(ang) if kind < 2 else torch.sin(ang))
    if kind == 1:
        out[:, 0] = 1.0
    if kind == 3:
        out[:, n - 1] = 1.0 - 2.0 * (torch.arange(n, device=dev) % 2).double()
    return out


class _Exact:
    """The r2r transforms of one grid."""

    def __init__(self, nx, ny, nz):
        self.n = (nx, ny, nz)
        self.mats = {}

    def m(self, kind, n):
        if (kind, n) not in self.mats:
            self.mats[kind, n] = _matrix(kind, n)
        return self.mats[kind, n]

    def r2r(self, a, kinds):
        nx, ny, nz = self.n
        a = a.reshape(nx * ny, nz) @ self.m(kinds[2], nz).T
        a = torch.matmul(self.m(kinds[1], ny), a.reshape(nx, ny, nz))
        return (self.m(kinds[0], nx) @ a.reshape(nx, ny * nz)).reshape(nx, ny, nz)

    def __call__(self, plan, a):
        return self.r2r(a, q.quasi.PLAN_KINDS[plan])


def _shift(a, axis, by):
    """a moved by `by` places along `axis`, zeros moving in: out[i] = a[i - by]."""
    out = torch.zeros_like(a)
    n = a.shape[axis]
    if by > 0:
        out.narrow(axis, by, n - by).copy_(a.narrow(axis, 0, n - by))
    else:
        out.narrow(axis, 0, n + by).copy_(a.narrow(axis, -by, n + by))
    return out


def _exact_steps(cfg, psi0, steps):
    """The state after `steps` steps from psi0 (quasi.cpp:875-2033, quasi-stb.cpp:983-1968)."""
    dev, stb = _device(), cfg.variant == 1
    nx, ny, nz = shape = (cfg.nx, cfg.ny, cfg.nz)
    tr = _Exact(*shape)
    dx = 2.0 * math.pi / (cfg.q0 * cfg.nw)
    idx = [torch.arange(n, device=dev, dtype=torch.float64).reshape([-1 if b == a else 1 for b in range(3)])
           for a, n in enumerate(shape)]
    Q = [math.pi * i / (dx * n) for i, n in zip(idx, shape)]
    S = [math.pi * (i + 1) / (dx * n) for i, n in zip(idx, shape)]
    ep, nu = -0.001 * cfg.ep_arg, cfg.nu_arg * (0.1 if stb else 1.0)
    rho_s = cfg.kp * cfg.amp + cfg.rho_0
    rho_m = cfg.rho_m if cfg.rho_m > 0 else rho_s / 2
    scale, dt, q0, al, be, ga = 0.125 / (nx * ny * nz), cfg.dt, cfg.q0, cfg.alpha, cfg.beta, cfg.gamma
    q2 = Q[0] ** 2 + Q[1] ** 2 + Q[2] ** 2
    alin = ep - al * (q0 ** 2 - q2) ** 2
    if stb:
        c1, c2 = 1.0 + dt / 2 * alin, 1.0 - dt / 2 * alin
    else:
        c1, c2 = 2.0 - dt * rho_m * alin, 1.5 - dt * rho_m * alin
    mix = [[S[b] if a == b else Q[b] for b in range(3)] for a in range(3)]   # wavenumbers on the grid of S_a
    mq = [m[0] ** 2 + m[1] ** 2 + m[2] ** 2 for m in mix]
    isine, sine = ("iSTx", "iSTy", "iSTz"), ("STx", "STy", "STz")
    grad = lambda f, a: -S[a] * _shift(f, a, -1)   # noqa: E731

    # plane "i - 1" of S_x as the rank-boundary exchange delivers it to v_y, v_z
    src = torch.arange(nx, device=dev) - 1
    n0 = nx // cfg.emulate_ranks
    for r in range(1, cfg.emulate_ranks):
        src[r * n0] = (r - 1) * n0

    psi = torch.from_numpy(psi0).to(dev)
    psiq = scale * tr("CT", psi)
    psi = tr("iCT", psiq)
    nl = tr("CT", be * psi ** 3 - ga * psi ** 5)
    psiq_old, psi_old = psiq, psi
    zero = torch.zeros_like(psi)
    divv, rhoq, rho_old = zero, zero, zero
    vel = [zero, zero, zero]
    for n in range(1, steps + 1):
        nl_old = nl
        g = [tr(isine[a], grad(psiq, a)) for a in range(3)]
        if stb:
            sh = tr("iCT", -alin * psiq)
            mu = sh - be * psi ** 3 + ga * psi ** 5
            s = [mu * g[a] for a in range(3)]
            dq = zero
            df, rho = zero, torch.ones_like(psi)
        else:
            dfq = al * (q0 ** 2 - q2) * psiq
            df, lap = tr("iCT", dfq), tr("iCT", -q2 * dfq)
            rd = [tr(isine[a], grad(rhoq, a)) for a in range(3)]
            rho = cfg.kp * torch.sqrt(q0 ** 2 * psi ** 2 + g[0] ** 2 + g[1] ** 2 + g[2] ** 2) + cfg.rho_0
            rhoq = scale * tr("CT", rho) * torch.exp(-1.57 * 1.57 * 8 * q2)
            rho = tr("iCT", rhoq)
            if n > cfg.divv_switch:
                divv = -((rho - rho_old) / dt + vel[0] * rd[0] + vel[1] * rd[1] + vel[2] * rd[2]) / (
                    0.5 * (rho + rho_old))
            rho_old = rho
            dq = tr("CT", divv)
            lap = rho * lap
            s = [lap * g[a] - rho * df * tr(isine[a], -mq[a] * grad(psiq, a)) for a in range(3)]
        sq = [tr(sine[a], s[a]) for a in range(3)]
        back = [_shift(sq[a], a, 1) for a in range(3)]
        pq = -(Q[0] * back[0] + Q[1] * back[1] + Q[2] * back[2]) / q2
        if stb:
            pq = torch.where(idx[0] * idx[1] * idx[2] > 0, scale * (pq + nu * dq), zero)
        else:
            pq = torch.where(q2 > 0, scale * pq, zero)
        halo = torch.where(idx[0] > 0, sq[0][src.clamp(min=0)], zero)
        for a in range(3):
            comp = []
            for b in range(3):
                f = sq[b] if a == b else back[b] if b or not a else halo
                comp.append(f if a == b else _shift(f, a, -1))
            dot = sum(mix[a][b] * comp[b] for b in range(3))
            v = scale / (nu * mq[a]) * (comp[a] - S[a] / mq[a] * dot + nu * S[a] * _shift(dq, a, -1))
            if a == 0:
                v[nx - 1] = 0
            else:
                v[:, ny - 1] = 0
                v[:, :, nz - 1] = 0
            vel[a] = tr(isine[a], v)
        adv = vel[0] * g[0] + vel[1] * g[1] + vel[2] * g[2]
        if stb:
            nlr = be * psi ** 3 - ga * psi ** 5 - adv
        else:
            divv = tr("iCT", scale * dq)
            nlr = rho * (ep * psi - df + be * psi ** 3 - ga * psi ** 5) - lap - adv
            if n > cfg.divv_switch + 1:
                nlr = nlr + tr("iCT", pq) * cfg.kp / rho_s ** 2 * torch.sqrt(rd[0] ** 2 + rd[1] ** 2 + rd[2] ** 2)
        nl = tr("CT", nlr)
        if n == 1:
            nl_old = nl
        force = dt / 2 * scale * (3.0 * nl - nl_old)
        new = (c1 * psiq + force if stb else c1 * psiq - 0.5 * psiq_old + force) / c2
        psiq_old, psiq = psiq, new
        psi_old, psi = psi, tr("iCT", psiq)
    dx3 = dx ** 3
    energy = float((rho * (-0.5 * ep * psi ** 2 + 0.5 * al * df ** 2 - 0.25 * be * psi ** 4
                           + ga / 6 * psi ** 6)).sum()) * dx3
    i, k = round(cfg.q_pert * dx * nz / math.pi), round(cfg.q0 * dx * nz / math.pi)
    growth = float("nan")
    if i < nx and k < nz:
        a, b = float(psiq[i, 0, k]), float(psiq_old[i, 0, k])
        growth = (a - b) / (dt * b) if b else float("nan")
    return {"psi": psi.cpu().numpy(), "rho": rho.cpu().numpy(), "vz": vel[2].cpu().numpy(), "growth": growth,
            "L1": float((psi - psi_old).abs().sum() / (dt * psi.abs().sum())),
            "mass": float(rho.sum()) * dx3, "energy": 0.0 if stb else energy}


def exact(case, seed):
    c = case
    if c["kind"] == "r2r":
        x = _field_in(c, seed).double().to(_device())
        return _Exact(c["nx"], c["ny"], c["nz"])(c["plan"], x)
    if c["kind"] == "step":
        cfg = _config(c)
        e = _exact_steps(cfg, _initial(c, cfg, seed), c["steps"])
        return {k: e[k] for k in _outputs(c)}
    cfgs, psis = _member_setup(c, seed)
    es = [_exact_steps(cfg, psi, c["steps"]) for cfg, psi in zip(cfgs, psis)]
    return {"growth": np.array([e["growth"] for e in es]), "psi": [e["psi"] for e in es]}
