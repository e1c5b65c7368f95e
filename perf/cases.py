"""What the speed of this framework is measured on: the calls a user makes, over the
sizes, storage forms and options those calls are made with.

Lattice-Boltzmann cases are solver contexts on the repository's seeded vessel
generators, started from a smooth seeded flow field; one pass steps them the way a
program does (plain steps, graph steps, steps with the StabilityTester, a run
towards steady state, a read of the fields) and returns the whole state.  Network
cases are the warm-start surrogate's calls: a training step, a prediction, one
convolution layer forward and backward.

``exact`` gives the same results in 64 bits from plain numpy / torch: its own site
numbering, neighbour search, collision and link rules, and convolutions as shifted
matrix products.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from hemelb_gb300 import capi, cases, surrogate

PRECISION = {"fp64": capi.FP64, "fp32": capi.FP32DEV, "fp16": capi.FP16}
ELEM = {"fp64": 8, "fp32": 4, "fp16": 2}
Q = 19


def listed():
    return [
        # Straight pipe, 25k sites: the smallest geometry of the test-suite, a few
        # steps at a time (coupled or scripted runs); launch latency counts.
        {"name": "pipe_fp64", "vessel": "pipe", "radius": 10.0, "length": 80, "precision": "fp64",
         "mode": "step", "steps": 10, "autotune": False},
        # Bifurcation, 1.5M sites, BFL walls and a pulsatile Ladd inlet in the plain
        # FP64 form: the reference's own arithmetic, as a user of it starts out.
        {"name": "bifurcation_fp64", "vessel": "bifurcation", "radius": 24.0, "length": 200.0, "factor": 2.5,
         "geometry_seed": 1234, "precision": "fp64", "mode": "step", "steps": 10, "autotune": False},
        # One vessel of the warm start's data generation: a small FP64 geometry run
        # towards steady state, checked after every step, and its fields read back.
        {"name": "vessel_steady_fp64", "vessel": "box", "box": 96, "kind": 1, "geometry_seed": 11, "tau": 0.8,
         "drho": 1.5e-3, "precision": "fp64", "mode": "steady", "steps": 500, "autotune": False},
        # The bifurcation with FP32 deviations, replayed as a graph.
        {"name": "bifurcation_fp32", "vessel": "bifurcation", "radius": 24.0, "length": 200.0, "factor": 2.5,
         "geometry_seed": 1234, "precision": "fp32", "mode": "graph", "steps": 20, "autotune": False},
        # Vascular tree, 16.9M sites, TRT: the benchmark's generator and physics at a
        # size whose distributions are far larger than L2 (the largest update).
        {"name": "tree_fp32", "vessel": "tree", "box": 512, "roots": 1, "depth": 6, "radius": 50.0,
         "geometry_seed": 7, "precision": "fp32", "mode": "step", "steps": 20, "autotune": True},
        # The same solver as a monitored simulation: one call per step, the
        # StabilityTester on a 6-step cadence.
        {"name": "tree_fp32_monitored", "vessel": "tree", "box": 384, "roots": 2, "depth": 6, "radius": 32.0,
         "geometry_seed": 7, "precision": "fp32", "mode": "monitored", "steps": 12, "interval": 6,
         "autotune": True},
        # Half-size storage for the same kind of tree.
        {"name": "tree_fp16", "vessel": "tree", "box": 384, "roots": 2, "depth": 6, "radius": 32.0,
         "geometry_seed": 7, "precision": "fp16", "mode": "step", "steps": 20, "autotune": True},
        # Batched ensemble of stenosed pipes (per-member tau, Ladd inlets) in one
        # context, graph steps: parameter studies.
        {"name": "ensemble_fp32", "vessel": "ensemble", "members": 64, "geometry_seed": 2024, "precision": "fp32",
         "mode": "graph", "steps": 20, "autotune": True},
        # Output of a run: density, velocity, iolet fluxes and the stability
        # reduction of the current state, on the host.
        {"name": "fields_fp32", "vessel": "bifurcation", "radius": 24.0, "length": 200.0, "factor": 2.5,
         "geometry_seed": 1234, "precision": "fp32", "mode": "fields", "steps": 0, "autotune": False},
        # One training step of the warm-start network at its own size and batch.
        {"name": "unet_train", "net": "unet", "box": 96, "batch": 4, "train": True},
        # One prediction: the network on a single vessel, before a warm-started run.
        {"name": "unet_predict", "net": "unet", "box": 96, "batch": 1, "train": False},
        # One convolution layer forward and backward on a ragged volume.
        {"name": "conv_ragged", "net": "conv", "n": 1, "d": 45, "h": 53, "w": 39, "cin": 144, "cout": 48,
         "taps": 27, "relu": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    what = rng.choice(["pipe", "bifurcation", "box", "tree", "ensemble", "unet", "conv", "conv"])
    if what == "unet":
        return {"net": "unet", "box": 8 * rng.randint(2, 12), "batch": rng.randint(1, 4),
                "train": rng.random() < 0.6}
    if what == "conv":
        while True:
            c = {"net": "conv", "n": rng.randint(1, 4), "d": round(_log(rng, 3, 96)), "h": round(_log(rng, 3, 96)),
                 "w": round(_log(rng, 3, 96)), "cin": 16 * rng.choice([1, 1, 2, 3, 4, 6, 9, 12, 18]),
                 "cout": 16 * rng.choice([1, 1, 2, 3, 4, 6, 9, 12]), "taps": 27, "relu": True}
            if _conv_flops(c) < 1.0e12:
                return c
    precision = rng.choice(["fp64", "fp32", "fp32", "fp16"])
    steps = rng.randint(1, 20)
    c = {"vessel": what, "geometry_seed": rng.randrange(1, 1 << 30), "precision": precision, "steps": steps,
         "mode": rng.choice(["step", "graph", "monitored", "fields"]), "autotune": rng.random() < 0.5}
    if what == "pipe":
        c.update(radius=round(_log(rng, 4.0, 20.0), 2), length=round(_log(rng, 17, 260)))
    elif what == "bifurcation":
        c.update(radius=round(_log(rng, 6.0, 24.0), 2), length=round(_log(rng, 30.0, 200.0), 1), factor=1.5)
    elif what == "box":
        c.update(box=96, kind=rng.randint(0, 1), tau=round(rng.uniform(0.7, 1.0), 3),
                 drho=round(rng.uniform(5e-4, 3e-3), 6), mode="steady", precision="fp64",
                 steps=rng.randint(60, 500), autotune=False)
    elif what == "tree":
        box = 8 * rng.randint(24, 48)
        c.update(box=box, roots=rng.randint(1, 2), depth=rng.randint(4, 6), radius=round(box / 12.0, 1))
    else:
        c.update(members=round(_log(rng, 2, 64)))
    if c["mode"] == "monitored":
        c["interval"] = rng.choice([1, 1, 2, 6])
    if c["mode"] == "fields":
        c["steps"] = 0
    return c


# ---------------------------------------------------------------------------
# lattice-Boltzmann cases
# ---------------------------------------------------------------------------
def _vessel_key(case):
    keys = ("vessel", "geometry_seed", "radius", "length", "factor", "box", "kind", "tau", "drho", "roots",
            "depth", "members", "precision")
    return tuple((k, case[k]) for k in keys if k in case)


@functools.lru_cache(maxsize=3)
def _vessel(key):
    """The geometry, physics and iolets a program loads before it makes a solver."""
    c = dict(key)
    p = PRECISION[c["precision"]]
    if c["vessel"] == "pipe":
        return cases.pipe(c["radius"], c["length"], precision=p)
    if c["vessel"] == "bifurcation":
        return cases.bifurcation(c["geometry_seed"], c["radius"], c["length"], c["factor"], precision=p)
    if c["vessel"] == "tree":
        return cases.tree(c["geometry_seed"], c["box"], c["roots"], c["depth"], c["radius"], precision=p)
    if c["vessel"] == "ensemble":
        return cases.ensemble(c["members"], c["geometry_seed"], precision=p)
    smp = surrogate.Sample(seed=c["geometry_seed"], kind=c["kind"], tau=c["tau"], drho=c["drho"], box=c["box"])
    v = smp.case()
    v.u_ref = smp.u_ref(v.geometry)
    return v


def _first_step(vessel):
    """A time inside the inlet's pulse."""
    io = list(vessel.inlets) + list(vessel.outlets)
    period = max([i.vel_period for i in io] or [0.0])
    return 1 + int(period) // 4


def _start(xyz, seed, speed):
    """A smooth flow: density and velocity at the sites `xyz` (N x 3, device)."""
    rng = np.random.default_rng(seed)
    x = xyz.to(torch.float64)
    v = []
    for _ in range(4):
        f = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
        for _ in range(3):
            k = torch.as_tensor(rng.uniform(-1, 1, 3) * 2 * np.pi / rng.uniform(30, 120), device=x.device)
            f += float(rng.uniform(0.3, 1.0)) * torch.sin(x @ k + float(rng.uniform(0, 6.28)))
        v.append(f / 3)
    rho = 1.0 + 0.05 * speed * v[0]
    return rho, speed * torch.stack(v[1:], dim=1)


def _speed(case, vessel):
    return 0.3 * vessel.u_ref if case["mode"] == "steady" else 0.01


def _prepare_vessel(case, seed):
    vessel = _vessel(_vessel_key(case))
    speed = _speed(case, vessel)
    if case["mode"] == "steady":
        runner = surrogate.SteadyRunner(vessel, vessel.u_ref, tol=1e-9)
        rho, u = _start(torch.as_tensor(runner.coords, device="cuda"), seed, speed)
        rho, u = rho.cpu().numpy(), u.cpu().numpy()
        return {"case": case, "runner": runner, "start": lambda coords: (rho, u)}
    s = vessel.solver()
    if case["autotune"]:
        s.SetInitialConditions()
        s.autotune(3)
    rho, u = _start(torch.as_tensor(s.site_coords(), device="cuda"), seed, speed)
    s.SetInitialField(rho.cpu().numpy(), u.cpu().numpy())
    s.SetTimeStep(_first_step(vessel))
    if case["mode"] == "monitored":
        s.SetMonitorInterval(case["interval"])
    f = torch.empty((s.n_sites, Q), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return {"case": case, "solver": s, "f": f}


def _run_vessel(state):
    case = state["case"]
    if case["mode"] == "steady":
        rec, rho, u = state["runner"].run(start=state["start"], average=True, max_steps=case["steps"], timed=False)
        return {"steps_run": rec["steps_run"], "status": rec["status"], "rho": rho, "u": u}
    s = state["solver"]
    if case["mode"] == "fields":
        rho, u = s.macro()
        return {"rho": rho, "u": u, "flux": s.IoletFlux(), "mass": s.reduce().mass}
    stats = None
    if case["mode"] == "step":
        s.DoTimeStep(case["steps"])
    elif case["mode"] == "graph":
        s.DoTimeStepGraph(case["steps"])
    else:
        for _ in range(case["steps"]):
            stats = s.StepMonitored(1)
    capi.check(capi.load().hlbg_get_f_device(s.ctx, state["f"].data_ptr(), 0), s.ctx)
    out = {"f": state["f"]}
    if stats is not None:
        out.update(mass=stats.mass, max_du=stats.max_du, min_f=stats.min_f, unstable=stats.unstable_sites,
                   time_step=stats.time_step)
    return out


# ---- the same in 64 bits ----------------------------------------------------
CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1]
INV = [0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _bits_of_blocks(mask):
    return np.unpackbits(np.ascontiguousarray(mask).view(np.uint8).reshape(-1, 64), axis=1,
                         bitorder="little").astype(bool)


class _Sites:
    """Sites of a sparse block geometry in contiguous order (collision type, Morton
    order of the blocks, order in the block), their links and their neighbours."""

    def __init__(self, g):
        fluid = _bits_of_blocks(g.fluid_mask)
        nb = fluid.shape[0]
        bc = g.block_coords.astype(np.int64)
        key = np.zeros(nb, dtype=np.int64)
        for k in range(16):
            for a in range(3):
                key |= ((bc[:, a] >> k) & 1) << (3 * k + 2 - a)
        rank = np.empty(nb, dtype=np.int64)
        rank[np.argsort(key, kind="stable")] = np.arange(nb)
        slot = np.flatnonzero(fluid.reshape(-1))
        wall, iolet = np.zeros(nb * 512, np.uint32), np.zeros(nb * 512, np.uint32)
        ioid, stype = np.full(nb * 512, -1, np.int32), np.ones(nb * 512, np.int8)
        row = np.full(nb * 512, -1, np.int32)
        wall[g.link_site], iolet[g.link_site] = g.wall_mask, g.iolet_mask
        ioid[g.link_site], stype[g.link_site] = g.iolet_id, g.site_type
        row[g.link_site] = np.arange(len(g.link_site), dtype=np.int32)
        w, t = wall[slot] != 0, stype[slot]
        ctype = np.where(t == 2, np.where(w, 4, 2), np.where(t == 3, np.where(w, 5, 3), np.where(w, 1, 0)))
        order = np.argsort((ctype.astype(np.int64) << 50) | (rank[slot >> 9] << 9) | (slot & 511), kind="stable")
        slot, self.ctype = slot[order], ctype[order]
        loc = slot & 511
        self.block = slot >> 9
        self.xyz = bc[self.block] * 8 + np.stack([loc >> 6, (loc >> 3) & 7, loc & 7], axis=1)
        self.wall, self.iolet, self.ioid, self.row = wall[slot], iolet[slot], ioid[slot], row[slot]
        self.cut = g.cut_distance
        # neighbours through a table of the blocks
        grid = np.full(tuple(int(b) + 2 for b in g.blocks), -1, np.int64)
        grid[bc[:, 0] + 1, bc[:, 1] + 1, bc[:, 2] + 1] = np.arange(nb)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev = dev
        site_of = torch.full((nb * 512 + 1,), -1, dtype=torch.int32, device=dev)
        site_of[torch.as_tensor(slot, device=dev)] = torch.arange(len(slot), dtype=torch.int32, device=dev)
        grid, x = torch.as_tensor(grid, device=dev), torch.as_tensor(self.xyz, device=dev)
        self.nbr = []
        for d in range(Q):
            y = x + torch.tensor([CX[d], CY[d], CZ[d]], device=dev)
            b = grid[(y[:, 0] >> 3) + 1, (y[:, 1] >> 3) + 1, (y[:, 2] >> 3) + 1]
            s = b * 512 + ((y[:, 0] & 7) * 8 + (y[:, 1] & 7)) * 8 + (y[:, 2] & 7)
            self.nbr.append(site_of[torch.where(b >= 0, s, torch.full_like(s, nb * 512))])


@functools.lru_cache(maxsize=1)
def _sites(key):
    return _Sites(_vessel(key).geometry)


def _feq(rho, m, d):
    cm = CX[d] * m[0] + CY[d] * m[1] + CZ[d] * m[2]
    return W[d] * (rho - 1.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / rho + 4.5 * cm * cm / rho + 3 * cm)


def _moments(f):
    return sum(f), [sum(c[d] * f[d] for d in range(Q) if c[d]) for c in (CX, CY, CZ)]


class _Plain:
    """The update in plain torch, 64 bits: f and the array it is pushed into."""

    def __init__(self, vessel, st):
        self.st, self.dev = st, st.dev
        self.trt = vessel.params.kernel == capi.KERNEL_TRT
        self.bfl = vessel.params.wall == capi.WALL_BFL
        tau = np.full(len(st.block), vessel.params.tau)
        if getattr(vessel, "block_tau", None) is not None:
            tau = vessel.block_tau[st.block]
        tau = torch.as_tensor(tau, device=self.dev)
        self.wp, self.wm = -1 / tau, -1 / (0.5 + (3 / 16) / (tau - 0.5))
        self.io = list(vessel.inlets) + list(vessel.outlets)
        n_in = len(vessel.inlets)
        can_io = st.ctype >= 2
        can_wall = np.isin(st.ctype, (1, 4, 5))
        T = lambda a: torch.as_tensor(a, device=self.dev)
        self.links = []
        for d in range(Q):
            bit = lambda m, e: ((m >> np.uint32(e - 1)) & 1).astype(bool) if e else np.zeros(len(m), bool)
            io = can_io & bit(st.iolet, d)
            wall = can_wall & bit(st.wall, d) & ~io
            push = ~io & ~wall & (st.nbr[d].cpu().numpy() >= 0)
            e = {"push": T(np.flatnonzero(push))}
            e["to"] = st.nbr[d][e["push"]].long()
            w = np.flatnonzero(wall)
            if self.bfl and len(w):
                q = st.cut[st.row[w], d - 1].astype(np.float64)
                back = bit(st.wall, INV[d])[w]
                e["bounce"], e["bfl"] = T(w[back | (q < 0.5)]), T(w[~(back | (q < 0.5))])
                e["bfl_q"] = T(q[~(back | (q < 0.5))])
                e["post"], e["post_q"] = T(w[~back & (q < 0.5)]), T(q[~back & (q < 0.5)])
            else:
                e["bounce"] = T(w)
            i = np.flatnonzero(io)
            e["io"] = T(i)
            e["io_id"] = T(np.where(np.isin(st.ctype[i], (2, 4)), st.ioid[i], n_in + st.ioid[i]).astype(np.int64))
            self.links.append(e)
        self.xyz = T(st.xyz)
        n = [np.array(i.normal[:]) / np.linalg.norm(i.normal[:]) for i in self.io]
        self.n = T(np.array(n).reshape(-1, 3))
        self.nf = self.n.float().double()
        self.pos = T(np.array([i.position[:] for i in self.io]).reshape(-1, 3))
        self.radius = T(np.array([i.radius for i in self.io]))

    def start(self, rho, u):
        m = [rho * u[:, k] for k in range(3)]
        self.f = [_feq(rho, m, d) for d in range(Q)]
        self.g = [f.clone() for f in self.f]

    def step(self, t):
        """One step; t is the 1-indexed step."""
        f, g = self.f, self.g
        rho, m = _moments(f)
        eq = [_feq(rho, m, d) for d in range(Q)]
        if self.trt:
            post = [f[0] + self.wp * (f[0] - eq[0])]
            for d in range(1, Q, 2):
                a, b = f[d] - eq[d], f[d + 1] - eq[d + 1]
                s, o = 0.5 * self.wp * (a + b), 0.5 * self.wm * (a - b)
                post += [f[d] + s + o, f[d + 1] + s - o]
        else:
            post = [f[d] + self.wp * (f[d] - eq[d]) for d in range(Q)]
        dens, peak = [], []
        for i in self.io:
            nash = i.model == capi.IOLET_COSINE
            dens.append(i.density_mean + i.density_amp * math.cos(2 * math.pi / i.period * (t - 1) + i.phase)
                        if nash else 1.0)
            p = i.max_speed
            if i.model == capi.IOLET_PULSATILE:
                p *= 0.5 * (1 - math.cos(2 * math.pi * t / i.vel_period))
            peak.append(p)
        dens, peak = (torch.tensor(v, dtype=torch.float64, device=self.dev) for v in (dens, peak))
        nash = torch.tensor([i.model == capi.IOLET_COSINE for i in self.io], device=self.dev)
        for d in range(Q):
            e, inv = self.links[d], INV[d]
            g[d][e["to"]] = post[d][e["push"]]
            if d == 0:
                continue
            g[inv][e["bounce"]] = post[d][e["bounce"]]
            if "bfl" in e:
                s, q = e["bfl"], e["bfl_q"]
                g[inv][s] = (post[d][s] + (2 * q - 1) * post[inv][s]) / (2 * q)
            s, k = e["io"], e["io_id"]
            if s.numel():
                r = rho[s]
                ms = torch.stack([v[s] for v in m], dim=1)
                comp = (ms * self.nf[k]).sum(1) / r * dens[k]
                gm = [self.nf[k][:, a] * comp for a in range(3)]
                c = torch.tensor([CX[d], CY[d], CZ[d]], dtype=torch.float64, device=self.dev)
                h = self.xyz[s].double() + 0.5 * c - self.pos[k]
                z = (h * self.n[k]).sum(1)
                sp = peak[k] * (1 - ((h * h).sum(1) - z * z) / (self.radius[k] ** 2).clamp(min=1e-300)) * r
                ladd = post[d][s] - 6 * W[d] * (self.n[k] @ c) * sp
                g[inv][s] = torch.where(nash[k], _feq(dens[k], gm, inv), ladd)
        for d in range(1, Q):
            e, inv = self.links[d], INV[d]
            if "post" in e:
                s, q = e["post"], e["post_q"]
                g[inv][s] = 2 * q * g[inv][s] + (1 - 2 * q) * g[d][s]
        self.f, self.g = g, f

    def velocity(self, f):
        rho, m = _moments(f)
        return rho, torch.stack([v / rho for v in m], dim=1)


def _exact_vessel(case, seed):
    vessel = _vessel(_vessel_key(case))
    if vessel.geometry.n_fluid * (case["steps"] + 2) > 1.0e9:
        return None
    st = _sites(_vessel_key(case))
    p = _Plain(vessel, st)
    p.start(*_start(p.xyz, seed, _speed(case, vessel)))
    if case["mode"] == "steady":
        p.step(1)
        p.f = [0.5 * (a + b) for a, b in zip(p.f, p.g)]
        for k in range(case["steps"]):
            p.step(2 + k)
        rho, u = p.velocity(p.f)
        return {"steps_run": None, "status": None, "rho": rho, "u": u}
    t = _first_step(vessel)
    if case["mode"] == "fields":
        rho, u = p.velocity(p.f)
        flux = torch.zeros(len(p.io), dtype=torch.float64, device=p.dev)
        n_in = len(vessel.inlets)
        s = np.flatnonzero((st.ctype >= 2) & (st.ioid >= 0))
        k = torch.as_tensor(np.where(np.isin(st.ctype[s], (2, 4)), st.ioid[s], n_in + st.ioid[s]).astype(np.int64),
                            device=p.dev)
        s = torch.as_tensor(s, device=p.dev)
        flux.index_add_(0, k, ((rho[:, None] * u)[s] * p.n[k]).sum(1))
        return {"rho": rho, "u": u, "flux": flux, "mass": rho.sum()}
    out, before = {}, None
    for k in range(case["steps"]):
        if case["mode"] == "monitored" and (t + k) % case["interval"] == 0 and before is not None:
            # the check of this step: the state it collides against the one before
            rho, u = p.velocity(p.f)
            out = {"mass": rho.sum(), "max_du": (u - p.velocity(before)[1]).norm(dim=1).max(),
                   "min_f": min(v.min() for v in p.f)}
        before = p.f
        p.step(t + k)
        if case["mode"] == "monitored":
            before = [v.clone() for v in before]
    none = {"mass": None, "max_du": None, "min_f": None, "unstable": None, "time_step": None}
    out = {**none, **out} if case["mode"] == "monitored" else {}
    return {"f": torch.stack(p.f, dim=1), **out}


# ---------------------------------------------------------------------------
# network cases
# ---------------------------------------------------------------------------
def _conv_flops(c):
    return 3 * 2.0 * c["taps"] * c["cin"] * c["cout"] * c["n"] * c["d"] * c["h"] * c["w"]


def _tubes(n, box, gen):
    """Masks and signed distances of straight and bent tubes in n boxes."""
    ax = torch.arange(box, device="cuda", dtype=torch.float32) + 0.5
    x, y, z = torch.meshgrid(ax, ax, ax, indexing="ij")
    sd = []
    for _ in range(n):
        r, a, b, k = (torch.rand(4, generator=gen, device="cuda") * 2 - 1).tolist()
        cx = box * (0.5 + 0.15 * a * torch.sin(z * (6.28 / box) * (1 + 0.3 * k)))
        cy = box * (0.5 + 0.15 * b * torch.cos(z * (6.28 / box)))
        sd.append(box * (0.1 + 0.03 * r) - torch.sqrt((x - cx) ** 2 + (y - cy) ** 2))
    sd = torch.stack(sd)
    return (sd > 0).float(), (sd / 8).clamp(-2, 2), torch.stack([x, y, z], dim=-1) / box - 0.5


def _net_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, box = case["batch"], case["box"]
    mask, sd, pos = _tubes(n, box, gen)
    x = torch.zeros((n, box, box, box, 16), device="cuda")
    x[..., 0], x[..., 1], x[..., 4:7] = mask, sd, pos
    x[..., 2:4] = (torch.rand((n, 1, 1, 1, 2), generator=gen, device="cuda") * 2 - 1)
    t = torch.zeros((n, box, box, box, 16), device="cuda")
    t[..., :4] = mask[..., None] * torch.rand((n, 1, 1, 1, 4), generator=gen, device="cuda") * sd[..., None]
    return x.to(torch.bfloat16).contiguous(), t.contiguous(), mask.contiguous(), gen


def _prepare_unet(case, seed):
    x, target, mask, gen = _net_inputs(case, seed)
    net = surrogate.UNet(seed=seed)
    if case["train"]:  # moments as in the middle of a training run
        net.t = 1000
        for c in net.L.values():
            for m, v in ((c.mw, c.vw), (c.mb, c.vb)):
                m.copy_(torch.randn(m.shape, generator=gen, device="cuda") * 1e-4)
                v.copy_((torch.rand(v.shape, generator=gen, device="cuda") + 0.5) * 1e-6)
    return {"case": case, "net": net, "x": x, "target": target, "mask": mask}


def _run_unet(state):
    net = state["net"]
    out = net.forward(state["x"])
    if not state["case"]["train"]:
        return {"out": out}
    dout = torch.empty(out.shape, dtype=torch.bfloat16, device=out.device)
    # the loss itself is a logged number, a sum in whatever order the GPU took
    surrogate.nn.mse(out, state["target"], state["mask"], dout)
    net.zero_grad()
    net.backward(dout)
    net.step(2e-5)
    L = net.L
    return {"out": out, "gw": [L[k].gw for k in net.NAMES], "gb": [L[k].gb for k in net.NAMES],
            "w": [L[k].w for k in net.NAMES], "b": [L[k].b for k in net.NAMES]}


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["n"], case["d"], case["h"], case["w"])
    x = torch.randn(shape + (case["cin"],), generator=gen, device="cuda").relu().to(torch.bfloat16)
    dy = (torch.randn(shape + (case["cout"],), generator=gen, device="cuda") * 1e-3).to(torch.bfloat16)
    return x.contiguous(), dy.contiguous()


def _prepare_conv(case, seed):
    x, dy = _conv_inputs(case, seed)
    layer = surrogate.Conv(case["cin"], case["cout"], np.random.default_rng(seed), taps=case["taps"],
                           relu=case["relu"])
    return {"case": case, "layer": layer, "x": x, "dy": dy}


def _run_conv(state):
    layer = state["layer"]
    layer.zero_grad()
    y = layer.forward(state["x"])
    dx = layer.backward(state["dy"])
    return {"y": y, "dx": dx, "gw": layer.gw, "gb": layer.gb}


def _windows(a, b, dz, dy, dx):
    """Views of `a` (read at the voxel shifted by the offset) and `b` (at the voxel)."""
    def cut(n, o):
        return slice(max(0, o), n + min(0, o)), slice(max(0, -o), n + min(0, -o))
    (za, zb), (ya, yb), (xa, xb) = (cut(a.shape[k + 1], o) for k, o in enumerate((dz, dy, dx)))
    return a[:, za, ya, xa], b[:, zb, yb, xb]


def _offsets(taps):
    return [(t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1) for t in range(27)] if taps == 27 else [(0, 0, 0)]


class _PlainConv:
    def __init__(self, w, b, taps, relu):
        self.w, self.b, self.taps, self.relu = w.to(torch.bfloat16).double(), b.double(), taps, relu

    def forward(self, x):
        y = self.b.expand(tuple(x.shape[:4]) + (len(self.b),)).clone()
        for t, o in enumerate(_offsets(self.taps)):
            a, v = _windows(x, y, *o)
            v += a @ self.w[t].T
        self.x, self.y = x, y.relu() if self.relu else y
        return self.y

    def backward(self, dy, need_dx=True):
        if self.relu:
            dy = dy * (self.y > 0)
        self.gb = dy.sum((0, 1, 2, 3))
        self.gw = torch.zeros_like(self.w)
        dx = torch.zeros_like(self.x) if need_dx else None
        for t, o in enumerate(_offsets(self.taps)):
            a, g = _windows(self.x, dy, *o)
            self.gw[t] = g.reshape(-1, g.shape[-1]).T @ a.reshape(-1, a.shape[-1])
            if need_dx:
                _windows(dx, dy, *o)[0].add_(g @ self.w[t])
        self.x = self.y = None
        return dx


def _pool(x):
    n, d, h, w, c = x.shape
    return x.view(n, d // 2, 2, h // 2, 2, w // 2, 2, c).mean((2, 4, 6))


def _spread(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


def _exact_unet(case, seed):
    if case["train"] and case["batch"] * case["box"] ** 3 > 2 * 96 ** 3:
        return None  # over 20 s in 64 bits
    st = _prepare_unet(case, seed)
    net = st["net"]
    L = {k: _PlainConv(c.w, c.b, c.taps, c.relu) for k, c in net.L.items()}
    run = lambda names, x: functools.reduce(lambda v, k: L[k].forward(v), names, x)
    e0 = run(("e0a", "e0b"), st["x"].double())
    e1 = run(("e1a", "e1b"), _pool(e0))
    e2 = run(("e2a", "e2b"), _pool(e1))
    b = run(("ba", "bb"), _pool(e2))
    d2 = run(("d2a", "d2b"), torch.cat([_spread(b), e2], -1))
    d1 = run(("d1a", "d1b"), torch.cat([_spread(d2), e1], -1))
    d0 = run(("d0a", "d0b"), torch.cat([_spread(d1), e0], -1))
    out = L["head"].forward(d0)
    if not case["train"]:
        return {"out": out}
    m = st["mask"][..., None].double()
    g = 2 * m * (out - st["target"].double()) / max(float(m.sum()) * out.shape[-1], 1.0)
    back = lambda names, v, **kw: functools.reduce(lambda a, k: L[k].backward(a), names, v)
    g = back(("head", "d0b", "d0a"), g)
    c = d1.shape[-1]
    ge0, g = g[..., c:], 8 * _pool(g[..., :c])
    g = back(("d1b", "d1a"), g)
    c = d2.shape[-1]
    ge1, g = g[..., c:], 8 * _pool(g[..., :c])
    g = back(("d2b", "d2a"), g)
    c = b.shape[-1]
    ge2, g = g[..., c:], 8 * _pool(g[..., :c])
    g = back(("bb", "ba"), g)
    g = back(("e2b", "e2a"), ge2 + _spread(g) / 8)
    g = back(("e1b", "e1a"), ge1 + _spread(g) / 8)
    g = L["e0b"].backward(ge0 + _spread(g) / 8)
    L["e0a"].backward(g, need_dx=False)
    res = {"out": out, "gw": [], "gb": [], "w": [], "b": []}
    t = net.t + 1
    for k in net.NAMES:
        p, c = L[k], net.L[k]
        res["gw"].append(p.gw)
        res["gb"].append(p.gb)
        for name, w, g, mm, v in (("w", c.w, p.gw, c.mw, c.vw), ("b", c.b, p.gb, c.mb, c.vb)):
            mm, v = 0.9 * mm.double() + 0.1 * g, 0.999 * v.double() + 0.001 * g * g
            res[name].append(w.double() - 2e-5 * (mm / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8))
    return res


def _exact_conv(case, seed):
    x, dy = _conv_inputs(case, seed)
    c = surrogate.Conv(case["cin"], case["cout"], np.random.default_rng(seed), taps=case["taps"],
                       relu=case["relu"])
    p = _PlainConv(c.w, c.b, case["taps"], case["relu"])
    y = p.forward(x.double())
    dx = p.backward(dy.double())
    return {"y": y, "dx": dx, "gw": p.gw, "gb": p.gb}


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if "vessel" in case:
        return _prepare_vessel(case, seed)
    return _prepare_unet(case, seed) if case["net"] == "unet" else _prepare_conv(case, seed)


def run(state):
    case = state["case"]
    if "vessel" in case:
        return _run_vessel(state)
    return _run_unet(state) if case["net"] == "unet" else _run_conv(state)


def exact(case, seed):
    if "vessel" in case:
        return _exact_vessel(case, seed)
    return _exact_unet(case, seed) if case["net"] == "unet" else _exact_conv(case, seed)


def work(case):
    if "vessel" in case:
        n, s = _vessel(_vessel_key(case)).geometry.n_fluid, ELEM[case["precision"]]
        if case["mode"] == "fields":
            return {"bytes": n * (3 * Q * s + 32), "flops": n * 200}
        # each step reads and writes every distribution once; then the state is read out
        out = 32 if case["mode"] == "steady" else 8 * Q
        return {"bytes": n * (case["steps"] * 2 * Q * s + Q * s + out), "flops": n * case["steps"] * 220}
    if case["net"] == "conv":
        m = case["n"] * case["d"] * case["h"] * case["w"]
        ci, co = case["cin"], case["cout"]
        # x and dy read, y and dx written; weights read, their gradient written
        return {"bytes": 2 * m * (2 * ci + 2 * co) + 6 * case["taps"] * ci * co, "flops": _conv_flops(case)}
    v0 = case["batch"] * case["box"] ** 3
    spec = ((1, ((16, 16), (16, 16), (64, 16), (16, 16))), (8, ((16, 48), (48, 48), (144, 48), (48, 48))),
            (64, ((48, 96), (96, 96), (288, 96), (96, 96))), (512, ((96, 192), (192, 192))))
    flops = sum(54.0 * ci * co * v0 / k for k, layers in spec for ci, co in layers) + 512.0 * v0
    act = sum(2.0 * (ci + co) * v0 / k for k, layers in spec for ci, co in layers)
    params = 3243024
    if case["train"]:  # forward, input gradient, weight gradient; Adam on the weights
        return {"bytes": 3 * act + params * 34 + 128 * v0, "flops": 3 * flops}
    return {"bytes": act + params * 2 + 64 * v0, "flops": flops}
