"""Measured workloads: what a program built on this library has it do.

A case is one frame of a simulation: put a saved state back into the scene
(Snapshot.restore, a checkpoint in device memory), advance `steps` time steps,
and read the state back, as `solve` does between two output frames.  The state
is saved a few steps after the start, so a pass can be repeated and gives the
same answer.

kinds
  sph      WCSPH dam break (nx x ny x nz fluid lattice in a tank of dummies)
  batch    several dam breaks of the scene stream stepped as one device scene
  drop     polydisperse spheres falling onto a plane (mostly free flight)
  bounce   equal spheres on a jittered lattice hitting a plane
  pack     touching spheres with friction, rolling and torsion springs
  beam     bonded cantilever beam beside rigid 3-sphere clumps
  coupled  DEM balls immersed in a tank of water, coupled particle by particle

`exact` restates each kind in FP64 on plain torch tensors.
"""
import math

import numpy as np
import torch

from this_studio_b200 import DEMSolver, DEMSPHCoupling, WCSPHSolver, batch, scenes


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the plain 4,096-sphere bounce, a short frame: launches and the host count
        {"name": "bounce_4096_mixed", "kind": "bounce", "side": 16, "precision": "mixed", "steps": 50},
        # the same spheres as a touching pack: contact history on every pair
        {"name": "pack_4096_mixed", "kind": "pack", "side": 16, "precision": "mixed", "steps": 100},
        # a larger pack in the reference's arithmetic
        {"name": "pack_64k_fp64", "kind": "pack", "side": 40, "precision": "fp64", "steps": 100},
        # a million spheres of the scene stream's DEM drop
        {"name": "drop_1m_mixed", "kind": "drop", "n": 1000000, "precision": "mixed", "steps": 200},
        # half the length of the bonded beam + clumps configuration
        {"name": "beam_110k_mixed", "kind": "beam", "nx": 200, "ny": 20, "clumps": 10000, "precision": "mixed",
         "steps": 100},
        # the smallest scene of the stream
        {"name": "sph_1k_mixed", "kind": "sph", "nx": 8, "ny": 8, "nz": 16, "dx": 0.01, "precision": "mixed",
         "steps": 100},
        # the size of the reference's own dam break, in its arithmetic
        {"name": "sph_18k_fp64", "kind": "sph", "nx": 21, "ny": 41, "nz": 21, "dx": 0.005, "precision": "fp64",
         "steps": 100},
        # the dam break configuration, mixed precision and FP64
        {"name": "sph_128k_mixed", "kind": "sph", "nx": 40, "ny": 40, "nz": 80, "dx": 0.01, "precision": "mixed",
         "steps": 100},
        {"name": "sph_128k_fp64", "kind": "sph", "nx": 40, "ny": 40, "nz": 80, "dx": 0.01, "precision": "fp64",
         "steps": 60},
        # the same tank at half the spacing
        {"name": "sph_1m_mixed", "kind": "sph", "nx": 80, "ny": 80, "nz": 160, "dx": 0.005, "precision": "mixed",
         "steps": 60},
        # eight dam breaks of uneven size as the server batches them
        {"name": "batch_8_mixed", "kind": "batch", "members": 8, "n_min": 1000, "n_max": 60000, "precision": "mixed",
         "steps": 100},
        # eight balls in a tank of water, two DEM substeps per fluid step
        {"name": "coupled_190k_mixed", "kind": "coupled", "nx": 64, "depth": 48, "balls": 8, "precision": "mixed",
         "steps": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sph", "sph", "sph", "batch", "drop", "drop", "bounce", "pack", "pack", "beam", "coupled"])
    c = {"kind": kind, "precision": rng.choice(["mixed", "mixed", "fp64"]), "steps": rng.choice([25, 50, 75, 100])}
    if kind == "sph":
        n = _log_int(rng, 1000, 500000)
        a, b = rng.uniform(0.6, 1.6), rng.uniform(0.8, 2.4)
        nx = max(4, int(round((n / (a * b)) ** (1.0 / 3.0))))
        c.update(nx=nx, ny=max(4, int(round(a * nx))), nz=max(6, int(round(b * nx))),
                 dx=rng.choice([0.004, 0.005, 0.01, 0.02]))
    elif kind == "batch":
        c.update(members=rng.randint(2, 12), n_min=1000, n_max=_log_int(rng, 4000, 60000))
    elif kind == "drop":
        c.update(n=_log_int(rng, 1000, 600000))
    elif kind == "bounce":
        c.update(side=_log_int(rng, 8, 60))
    elif kind == "pack":
        c.update(side=_log_int(rng, 8, 50))
    elif kind == "beam":
        c.update(nx=_log_int(rng, 20, 200), ny=rng.randint(4, 20), clumps=_log_int(rng, 50, 8000))
    else:
        c.update(nx=rng.randint(24, 60), depth=rng.randint(24, 44), balls=rng.randint(1, 8))
    return c


# ----------------------------------------------------------------- scenes --
def _flow(rng, x, speed):
    """A smooth velocity field with seeded phases and 2% noise."""
    ext = float(np.max(x.max(axis=0) - x.min(axis=0)))
    v = np.zeros_like(x)
    for k in range(3):
        for m in range(3):
            w = 2.0 * math.pi * rng.uniform(0.3, 1.2, 3) / ext
            v[:, k] += rng.uniform(0.3, 1.0) * np.sin(x @ w + rng.uniform(0, 2 * math.pi))
    v *= speed / max(1e-30, float(np.sqrt(np.mean(v * v))))
    return v + 0.02 * speed * rng.standard_normal(x.shape)


def _sph_scene(case, seed):
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    sc = scenes.sph_dam_break(nx, ny, nz, dx, tank=(4 * nx * dx, ny * dx, (nz + nz // 4) * dx),
                              column_height=nz * dx)
    rng = np.random.default_rng(seed)
    sc.fluid = sc.fluid + rng.uniform(-0.1 * dx, 0.1 * dx, sc.fluid.shape)
    sc.velocity = _flow(rng, sc.fluid, 0.15 * math.sqrt(9.81 * nz * dx))
    return sc


def _batch_scenes(case, seed):
    rng = np.random.default_rng(seed)
    c0 = 10.0 * math.sqrt(2 * 9.81 * 0.01 * 2 * (case["n_max"] / 2.0) ** (1.0 / 3.0))
    dt = 0.25 * 0.013 / (1.2 * c0)
    out = []
    for n in np.geomspace(case["n_min"], case["n_max"], case["members"]):
        sc = scenes.sph_column(int(n), c0, dt)
        sc.fluid = sc.fluid + rng.uniform(-0.1 * sc.spacing, 0.1 * sc.spacing, sc.fluid.shape)
        out.append(sc)
    return out


def _dem_scene(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "bounce":
        sc = scenes.dem_drop(n_side=case["side"], seed=seed, plane_gap=0.0)
    elif case["kind"] == "drop":
        sc = scenes.dem_drop_poly(case["n"], seed=seed)
        sc.position[:, 2] -= 0.1 * 0.005 * math.sqrt(3.0)  # the lowest sphere touches the plane
    elif case["kind"] == "pack":
        return scenes.dem_pack(n_side=case["side"], seed=seed)
    else:
        return scenes.bonded_beam_clumps(nx=case["nx"], ny=case["ny"], nz=case["ny"], n_clumps=case["clumps"],
                                         seed=seed)
    sc.velocity = rng.normal(0.0, 0.1, sc.position.shape) + np.array([0.0, 0.0, -1.0])
    return sc


def _coupled_scene(case, seed):
    rng = np.random.default_rng(seed)
    balls = []
    for k in range(case["balls"]):
        at = [(0.25, 0.75)[k >> s & 1] for s in range(2)] + [(0.35, 0.75)[k >> 2 & 1]]
        balls.append((at[0], at[1], at[2], 5.0, rng.uniform(500.0, 2500.0)))
    return scenes.balls_in_tank(nx=case["nx"], ny=case["nx"], depth=case["depth"], balls=balls, dem_substeps=2,
                                ball_velocity=rng.normal(0.0, 0.3, (len(balls), 3)))


def _build_sph(sc, precision):
    s = WCSPHSolver()
    s.addSPHs(sc.fluid, getattr(sc, "velocity", None), sc.sound_speed, sc.spacing, sc.density, sc.viscosity)
    s.addDummies(sc.dummy, None, sc.sound_speed, sc.spacing, sc.density, sc.viscosity)
    s.initialize(sc.minb, sc.maxb, sc.gravity, sc.dt, precision)
    return s


WARM = 10  # steps before the saved state: two re-sort periods of the DEM lists


def prepare(case, seed):
    if case["kind"] == "sph":
        s = _build_sph(_sph_scene(case, seed), case["precision"])
        for _ in range(2):  # the lists take their size after the first steps
            s.step(WARM // 2)
            s.synchronize()
        return {"case": case, "sph": s, "saved": [s.snapshot()]}
    if case["kind"] == "batch":
        b = batch.SPHBatch(case["precision"])
        b.members = [batch.Member(k, sc) for k, sc in enumerate(_batch_scenes(case, seed))]
        b.rebuild()
        for _ in range(2):
            b.step(WARM // 2)
        return {"case": case, "batch": b, "saved": [b.solver.snapshot()]}
    if case["kind"] == "coupled":
        f, d, c = scenes.build_coupled(_coupled_scene(case, seed), case["precision"])
        for _ in range(2):
            c.step(WARM // 2, 2)
        return {"case": case, "sph": f, "dem": d, "coupling": c, "saved": [f.snapshot(), d.snapshot()]}
    d = scenes.build_dem(_dem_scene(case, seed), case["precision"])
    d.step(WARM)
    return {"case": case, "dem": d, "saved": [d.snapshot()]}


_FLUID = ("position", "velocity", "acceleration", "density", "pressure", "densityChange")


def run(state):
    case = state["case"]
    for s in state["saved"]:
        s.restore()
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        b.capture()
        return [{k: m.state[k] for k in ("position", "velocity", "density", "pressure", "densityChange")}
                for m in b.members]
    if case["kind"] == "coupled":
        state["coupling"].step(case["steps"], 2)
        _, force, torque = state["coupling"].getForces()
        fluid = state["sph"].getSPH()
        return {"fluid": {k: fluid[k] for k in _FLUID}, "balls": state["dem"].getBall(), "force": force,
                "torque": torque}
    if case["kind"] == "sph":
        state["sph"].step(case["steps"])
        fluid = state["sph"].getSPH()
        return {k: fluid[k] for k in _FLUID}
    d = state["dem"]
    d.step(case["steps"])
    out = {"balls": d.getBall()}
    if case["kind"] == "beam":
        out["clumps"] = d.getClump()
        bonds = d.getBondedInteraction()
        out["bonds"] = {k: bonds[k] for k in ("isBonded", "normalForce", "shearForce", "bendingTorque")}
    return out


# ---------------------------------------------------------- work, tolerance --
def _counts(case):
    """(fluid, dummies, balls, contacts or bonds) of a case."""
    k = case["kind"]
    if k in ("sph", "coupled"):
        if k == "sph":
            nx, ny, nz, tall = case["nx"], case["ny"], case["nz"], case["nz"] // 4
            lx = 4 * nx
        else:
            nx = ny = lx = case["nx"]
            nz, tall = case["depth"], 12
        tank = lx * ny * (nz + tall)
        return nx * ny * nz, (lx + 6) * (ny + 6) * (nz + tall + 3) - tank, case.get("balls", 0), 0
    if k == "batch":
        f = d = 0
        for n in np.geomspace(case["n_min"], case["n_max"], case["members"]):
            nx = max(2, int(round((int(n) / 2.0) ** (1.0 / 3.0))))
            h = int(2.5 * nx)
            f += 2 * nx ** 3
            d += (4 * nx + 6) * (nx + 6) * (h + 3) - 4 * nx * nx * h
        return f, d, 0, 0
    if k == "beam":
        n = case["nx"] * case["ny"] ** 2
        return 0, 0, n + 3 * case["clumps"], 3 * n
    n = case["n"] if k == "drop" else case["side"] ** 3
    return 0, 0, n, 3 * n if k == "pack" else 0


def work(case):
    f, d, b, c = _counts(case)
    # a fluid particle's state (x, v, density change) read and written once a
    # step, a dummy's (x, normal) read once; a ball's (x, v, w) likewise, and a
    # contact's springs or a bond's state (9 values) read and written
    per_step = f * 14 * 8 + d * 6 * 8 + b * 18 * 8 + c * 18 * 8
    out = (f * 12 + b * 15) * 8
    # three passes of about 40 operations over some 75 neighbours; two force
    # evaluations of about 300 operations per contact and 60 per ball
    flops = f * 75 * 3 * 40 + 2 * (c * 300 + b * 60)
    return {"bytes": per_step * case["steps"] + out, "flops": flops * case["steps"]}


def tolerance(case):
    # against `exact` a frame's worst output is off by up to 3e-11 in FP64 (bond
    # torques near zero) and 2e-6 in mixed precision (a ball's spin in water);
    # a bond at its strength may break a step earlier or later
    if case["precision"] == "fp64":
        return {"rel": 2e-10, "max": 1e-6, "differ": 1e-4}
    return {"rel": 1e-5, "max": 1e-3, "differ": 1e-4}


# ------------------------------------------------------------ exact: shared --
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=_dev())


def _pairs(a, b, cut):
    """All (i, j) with |a_i - b_j| <= cut, sorted by i, by a cell search."""
    lo = torch.minimum(a.min(0).values, b.min(0).values) - cut
    ia, ib = ((a - lo) / cut).long(), ((b - lo) / cut).long()
    dim = torch.maximum(ia.max(0).values, ib.max(0).values) + 2
    key = (ib[:, 2] * dim[1] + ib[:, 1]) * dim[0] + ib[:, 0]
    key, order = torch.sort(key)
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            # three cells along x are one range of the sorted keys
            first = ((ia[:, 2] + dz) * dim[1] + ia[:, 1] + dy) * dim[0] + ia[:, 0] - 1
            s, e = torch.searchsorted(key, first), torch.searchsorted(key, first + 2, right=True)
            ok = (ia[:, 2] + dz >= 0) & (ia[:, 1] + dy >= 0)
            n = torch.where(ok, e - s, torch.zeros_like(s))
            for part in torch.arange(len(a), device=a.device).split(200000):
                m = n[part]
                i = torch.repeat_interleave(part, m)
                at = torch.arange(len(i), device=a.device) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
                j = order[s[i] + at]
                r = a[i] - b[j]
                hit = (r * r).sum(1) <= cut * cut
                found.append(torch.stack([i[hit], j[hit]]))
    p = torch.cat(found, 1)
    return p[:, torch.argsort(p[0], stable=True)]


def _rows(p, n):
    """Pairs sorted by i as padded rows: (the i that have pairs, j per row, -1 where none)."""
    cnt = torch.bincount(p[0], minlength=n)
    own = torch.nonzero(cnt).flatten()
    k = int(cnt.max()) if p.shape[1] else 0
    nb = torch.full((n, k), -1, dtype=torch.int64, device=p.device)
    at = torch.arange(p.shape[1], device=p.device) - (torch.cumsum(cnt, 0) - cnt)[p[0]]
    nb[p[0], at] = p[1]
    return own, nb[own]


def _dot(a, b):
    return (a * b).sum(-1)


# ------------------------------------------------------------- exact: fluid --
class _Fluid:
    """WCSPH in FP64 (Wendland C2, Riemann momentum and continuity, linear
    equation of state) on the neighbours of each step's start."""

    def __init__(self, sc):
        self.h, self.c, self.nu, self.rho0 = 1.3 * sc.spacing, sc.sound_speed, sc.viscosity, sc.density
        self.m = sc.spacing ** 3 * sc.density
        self.dt, self.g = sc.dt, _t(sc.gravity)
        self.x = _t(sc.fluid)
        v = getattr(sc, "velocity", None)
        self.v = torch.zeros_like(self.x) if v is None else _t(v)
        self.dr = torch.zeros(len(self.x), dtype=torch.float64, device=self.x.device)
        self.rho, self.p = self.dr + self.rho0, self.dr.clone()
        self.a = torch.zeros_like(self.x)
        # boundary particles: the dummies, and the markers of coupled balls
        d = _t(sc.dummy)
        own, nb = _rows(_pairs(d, d, 2 * self.h), len(d))
        n = torch.zeros_like(d)
        for rows, j in zip(own.split(65536), nb.split(65536)):
            r = d[rows][:, None] - d[j.clamp(min=0)]
            f, _, _ = self._kernel(r, (j >= 0) & (j != rows[:, None]))
            n[rows] = -(self.m / self.rho0) * (f[..., None] * r).sum(1)
        l = n.norm(dim=1, keepdim=True)
        self.bounds = [[d, torch.zeros_like(d), torch.where(l * l > 1e-10, n / l, torch.zeros_like(n))]]
        self.skin = 0.12 * 2 * self.h
        self.at = None

    def _kernel(self, r, keep):
        """gradW = f r, r_hat . gradW and 1 / r for pairs kept."""
        r2 = _dot(r, r)
        keep = keep & (r2 > 1e-40)
        inv = torch.where(keep, r2, torch.ones_like(r2)).rsqrt()
        q = r2 * inv / self.h
        t = (1.0 - 0.5 * q).clamp(min=0.0)
        w = 21.0 / (16.0 * math.pi * self.h ** 4) * 2.0 * t ** 3 * (t - 1.0 - 2.0 * q)
        w = torch.where(keep, w, torch.zeros_like(w))
        return w * inv, w, torch.where(keep, inv, torch.zeros_like(inv))

    def lists(self):
        """Candidate rows, renewed when something moved half the skin."""
        now = [self.x] + [b[0] for b in self.bounds]
        if self.at is not None and all(float(((a - b) ** 2).sum(1).max()) < (0.5 * self.skin) ** 2
                                       for a, b in zip(self.at, now)):
            return
        self.at = [a.clone() for a in now]
        cut = 2 * self.h + self.skin
        self.cand = []
        for k, b in enumerate(now):
            own, nb = _rows(_pairs(self.x, b, cut), len(self.x))
            step = 65536
            self.cand.append([(k, o, j) for o, j in zip(own.split(step), nb.split(step))])

    def neighbours(self):
        """This step's pairs: the candidates within the cutoff now."""
        self.lists()
        self.near = []
        for k, chunks in enumerate(self.cand):
            b = self.x if k == 0 else self.bounds[k - 1][0]
            for k, o, j in chunks:
                r = self.x[o][:, None] - b[j.clamp(min=0)]
                keep = (j >= 0) & (_dot(r, r) <= (2 * self.h) ** 2)
                if k == 0:
                    keep &= j != o[:, None]
                self.near.append((k, o, j.clamp(min=0), keep))

    def _boundary(self, o, j, b, r):
        """(v_j, n_j, extrapolated p, rho) of boundary neighbours."""
        P = self.p[o][:, None] + self.rho[o][:, None] * (-(r @ self.g)).clamp(min=0.0)
        return b[1][j], b[2][j], P, P / self.c ** 2 + self.rho0

    def accel(self, reaction=None):
        """Accelerations; `reaction` collects minus m a of each marker's term."""
        acc = torch.zeros_like(self.x)
        for k, o, j, keep in self.near:
            b = self.bounds[k - 1] if k else None
            r = self.x[o][:, None] - (b[0][j] if k else self.x[j])
            f, w, inv = self._kernel(r, keep)
            vi, rhoi, Pi = self.v[o][:, None], self.rho[o][:, None], self.p[o][:, None]
            if k == 0:
                vj, rhoj, Pj = self.v[j], self.rho[j], self.p[j]
                dU = -_dot(vi - vj, r) * inv
            else:
                vj, n, Pj, rhoj = self._boundary(o, j, b, r)
                dU = -2.0 * _dot(n, vi) + 2.0 * _dot(n, vj)
            beta = torch.minimum(3.0 * dU.clamp(min=0.0), torch.full_like(dU, self.c))
            Ps = 0.5 * (Pi + Pj) + 0.25 * beta * (rhoi + rhoj) * dU
            s = 2.0 * self.m / (rhoi * rhoj)
            term = (-(s * Ps * f))[..., None] * r + (s * self.nu * w)[..., None] * (vi - vj)
            acc[o] += term.sum(1)
            if reaction is not None and k == 2:
                reaction.index_add_(0, j[keep], -self.m * term[keep])
        return acc + self.g

    def density(self):
        s = torch.zeros_like(self.dr)
        for k, o, j, keep in self.near:
            b = self.bounds[k - 1] if k else None
            r = self.x[o][:, None] - (b[0][j] if k else self.x[j])
            f, w, inv = self._kernel(r, keep)
            vi, rhoi, Pi = self.v[o][:, None], self.rho[o][:, None], self.p[o][:, None]
            if k == 0:
                vj, rhoj, Pj = self.v[j], self.rho[j], self.p[j]
            else:
                vj, _, Pj, rhoj = self._boundary(o, j, b, r)
            X = (Pi - Pj) / (0.5 * (rhoi + rhoj) * self.c)
            s[o] += (self.m / rhoj * 0.5 * w * (_dot(vi - vj, r) * inv + X)).sum(1)
        self.dr = self.dr + self.dt * 2.0 * self.rho * s
        ch = self.dr.clamp(min=-0.1 * self.rho0)
        self.rho, self.p = ch + self.rho0, self.c ** 2 * ch

    def step(self, reaction=None):
        self.neighbours()
        self.a = self.accel(reaction)
        self.v = self.v + 0.5 * self.dt * self.a
        self.x = self.x + self.dt * self.v
        self.density()
        self.a = self.accel(reaction)
        self.v = self.v + 0.5 * self.dt * self.a

    def out(self, keys=_FLUID):
        got = dict(zip(_FLUID, (self.x, self.v, self.a, self.rho, self.p, self.dr)))
        return {k: got[k].cpu().numpy() for k in keys}


# ------------------------------------------------------------- exact: balls --
class _Balls:
    """DEM in FP64: Hertz-Mindlin contacts with springs, a plane of two
    triangles, parallel bonds and clumps, two force evaluations per step."""

    def __init__(self, sc):
        pos, vel = [sc.position], [np.zeros_like(sc.position) if sc.velocity is None else sc.velocity]
        rad, cl = [sc.radius], [np.full(len(sc.radius), -1)]
        m = 4.0 / 3.0 * math.pi * sc.radius ** 3 * sc.density
        fixed = np.zeros(len(m), bool) if sc.fixed is None else sc.fixed
        im = [np.where(fixed, 0.0, 1.0 / m)]
        w = getattr(sc, "angvel", None)
        self.nball = len(sc.position)
        for k, c in enumerate(sc.clumps):
            r = np.asarray(c["radius"], float)
            pos.append(c["point"])
            vel.append(np.tile(c["velocity"], (len(r), 1)))
            rad.append(r)
            cl.append(np.full(len(r), k))
            im.append(np.sum(r ** 3) / (c["mass"] * r ** 3))
        self.x, self.v, self.r, self.im = (_t(np.concatenate(a)) for a in (pos, vel, rad, im))
        self.w = torch.zeros_like(self.x)
        if w is not None:
            self.w[:self.nball] = _t(w)
        self.cl = torch.as_tensor(np.concatenate(cl), device=self.x.device)
        self.dt, self.g = sc.dt, _t(sc.gravity)
        _, _, E, G, e, krks, ktks, mus, mur, mut = sc.hertz[0]
        lr = math.log(e)
        self.E, self.G, self.D = E, G, -lr / math.sqrt(lr * lr + math.pi ** 2)
        self.kk, self.mu = (krks, ktks), (mus, mur, mut)
        # candidate pairs for the whole run: nothing closes this gap within it
        rmax = float(self.r.max())
        p = _pairs(self.x, self.x, 2.2 * rmax + 0.2 * rmax)
        p = p[:, p[0] < p[1]]
        gap = (self.x[p[0]] - self.x[p[1]]).norm(dim=1)
        ok = ~((self.im[p[0]] == 0) & (self.im[p[1]] == 0))
        ok &= ~((self.cl[p[0]] == self.cl[p[1]]) & (self.cl[p[0]] >= 0))
        near = ok & (gap <= 1.1 * (self.r[p[0]] + self.r[p[1]]))
        self.i, self.j = p[:, ok]
        self.sp = [torch.zeros(len(self.i), 3, dtype=torch.float64, device=self.x.device) for _ in range(3)]
        self.tri = None
        if sc.walls:
            self.tri = [_t(sc.walls[0]["vertices"])[[sc.walls[0][t][k] for t in ("tri0", "tri1", "tri2")]]
                        for k in range(2)]
            self.ws = torch.zeros(2, 3, len(self.x), 3, dtype=torch.float64, device=self.x.device)
        self.bonds = None
        if sc.bond_initial_contacts:
            b = p[:, near & (p[1] < self.nball)]
            n = self.x[b[0]] - self.x[b[1]]
            z = torch.zeros_like(n)
            _, _, gamma, Eb, knks, sigma, C, mu = sc.bonded[0]
            self.bpar = (gamma, Eb, knks, sigma, C, mu)
            self.bonds = {"b": b, "n": n / n.norm(dim=1, keepdim=True), "Fs": z, "Tb": z, "Fn": z[:, 0], "Tt": z[:, 0],
                          "ok": torch.ones(len(n), dtype=torch.bool, device=n.device)}
        self.fc = None
        if getattr(sc, "constant_force", None) is not None:
            self.fc = torch.zeros_like(self.x)
            self.fc[:self.nball] = _t(sc.constant_force)
        self.nc = len(sc.clumps)
        if self.nc:
            self.cx, self.cv, self.cw = (_t([c[k] for c in sc.clumps])
                                         for k in ("centroid", "velocity", "angularVelocity"))
            self.cim = 1.0 / _t([c["mass"] for c in sc.clumps])
            I = _t([[[c["inertia"][k] for k in row] for row in ((0, 3, 4), (3, 1, 5), (4, 5, 2))] for c in sc.clumps])
            self.cI = torch.linalg.inv(I)
            self.cq = torch.zeros(self.nc, 4, dtype=torch.float64, device=self.x.device)
            self.cq[:, 0] = 1.0
            self.peb = torch.nonzero(self.cl >= 0).flatten()
        self.extra = None  # held force and torque of a coupled fluid
        self.k = 0
        self.forces(0.0, 0.0)

    def _slide(self, s, sv, n, Fn, mu, k, c, dt):
        s1 = s - _dot(s, n)[:, None] * n
        a1 = s1.norm(dim=1, keepdim=True)
        s1 = torch.where(a1 > 1e-10, s1 * (s.norm(dim=1, keepdim=True) / a1.clamp(min=1e-300)), s1)
        return self._cap(s1 + sv * dt, sv, Fn, mu, k, c)

    def _cap(self, s, sv, Fn, mu, k, c):
        k, c = k[:, None], c[:, None]
        fs = -k * s - c * sv
        if mu > 0:
            af, an = fs.norm(dim=1, keepdim=True), Fn.norm(dim=1, keepdim=True)
            s = torch.where(af > mu * an, -(fs * (mu * an / af.clamp(min=1e-300)) + c * sv) / k.clamp(min=1e-300), s)
        return torch.where(k > 0, s, torch.zeros_like(s))

    def _law(self, sp, vc, wij, n, delta, m, R, dt):
        """Force, torque and springs of contacts with overlap delta > 0."""
        sq = (R * delta).sqrt()
        kn, ks = 4.0 / 3.0 * self.E * sq, 8.0 * self.G * sq
        k = (ks, ks * self.kk[0], ks * self.kk[1])
        z = 2.0 * math.sqrt(5.0 / 6.0) * self.D
        c = [z * (m * a).sqrt() for a in k]
        vn = _dot(vc, n)[:, None] * n
        Fn = (kn * delta)[:, None] * n - vn * (z * (m * kn).sqrt())[:, None]
        vs, R1 = vc - vn, R[:, None]
        s = self._slide(sp[0], vs, n, Fn, self.mu[0], k[0], c[0], dt)
        F = Fn - k[0][:, None] * s - c[0][:, None] * vs
        vr = -R1 * torch.linalg.cross(n, wij)
        sr = self._slide(sp[1], vr, n, Fn, self.mu[1], k[1], c[1], dt)
        T = R1 * torch.linalg.cross(n, -k[1][:, None] * sr - c[1][:, None] * vr)
        vt = 2.0 * R1 * _dot(wij, n)[:, None] * n
        st = _dot(sp[2] + vt * dt, n)[:, None] * n
        st = self._cap(st, vt, Fn, self.mu[2], k[2], c[2])
        T = T + 2.0 * R1 * (-k[2][:, None] * st - c[2][:, None] * vt)
        return F, T, (s, sr, st)

    def _contacts(self, F, T, dt):
        i, j = self.i, self.j
        d = self.x[i] - self.x[j]
        delta = self.r[i] + self.r[j] - d.norm(dim=1)
        on = torch.nonzero(delta > 0).flatten()
        old = [s[on] for s in self.sp]
        self.sp = [torch.zeros_like(s) for s in self.sp]
        if len(on) == 0:
            return
        i, j, d, delta = i[on], j[on], d[on], delta[on]
        n = d / d.norm(dim=1, keepdim=True)
        rc = self.x[j] + (self.r[j] - 0.5 * delta)[:, None] * n
        ai, aj = rc - self.x[i], rc - self.x[j]
        vc = self.v[i] + torch.linalg.cross(self.w[i], ai) - self.v[j] - torch.linalg.cross(self.w[j], aj)
        R = self.r[i] * self.r[j] / (self.r[i] + self.r[j])
        f, t, new = self._law(old, vc, self.w[i] - self.w[j], n, delta, 1.0 / (self.im[i] + self.im[j]), R, dt)
        for s, a in zip(self.sp, new):
            s[on] = a
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        T.index_add_(0, i, t + torch.linalg.cross(ai, f))
        T.index_add_(0, j, -t - torch.linalg.cross(aj, f))

    def _plane(self, F, T, dt):
        """The two triangles (0, 1, 3), (1, 2, 3) of a horizontal rectangle: the
        contact is the face below the centre; the other triangle's contact is
        on the shared edge and takes over the face's springs."""
        z = float(self.tri[0][0, 2])
        near = torch.nonzero(((self.x[:, 2] - z).abs() <= self.r) & (self.im > 0)).flatten()
        old = self.ws
        self.ws = torch.zeros_like(old)
        if len(near) == 0:
            return
        x, r = self.x[near], self.r[near]
        cp = x.clone()
        cp[:, 2] = z
        n = x - cp
        l = n.norm(dim=1)
        n = n / l[:, None]
        a, b = self.tri[0][1], self.tri[0][2]
        ab = b - a
        side = ab[0] * (x[:, 1] - a[1]) - ab[1] * (x[:, 0] - a[0])
        inner = ab[0] * (self.tri[0][0, 1] - a[1]) - ab[1] * (self.tri[0][0, 0] - a[0])
        face = torch.where(side * inner > 0, 0, 1)
        on_edge = a + (((x - a) @ ab) / (ab @ ab))[:, None] * ab
        other = _dot(x - on_edge, x - on_edge) <= r * r + 1e-12
        vc = self.v[near] + torch.linalg.cross(self.w[near], cp - x)
        sp = [old[face, k, near] for k in range(3)]
        f, t, new = self._law(sp, vc, self.w[near], n, r - l, 1.0 / self.im[near], r, dt)
        for k in range(3):
            self.ws[face, k, near] = new[k]
            self.ws[1 - face, k, near] = torch.where(other[:, None], sp[k], torch.zeros_like(sp[k]))
        F.index_add_(0, near, f)
        T.index_add_(0, near, t + torch.linalg.cross(cp - x, f))

    @staticmethod
    def _turn(v, ang):
        a = ang.norm(dim=1, keepdim=True)
        k = ang / a.clamp(min=1e-300)
        turned = (v * torch.cos(a) + torch.linalg.cross(k, v) * torch.sin(a) +
                  k * _dot(k, v)[:, None] * (1.0 - torch.cos(a)))
        return torch.where(a * a < 1e-20, v, turned)

    def _bonded(self, F, T, dt):
        B = self.bonds
        i, j = B["b"]
        gamma, Eb, knks, sigma, C, mu = self.bpar
        was = B["ok"]
        d = self.x[i] - self.x[j]
        l = d.norm(dim=1)
        n = d / l[:, None]
        delta = self.r[i] + self.r[j] - l
        rc = self.x[j] + (self.r[j] - 0.5 * delta)[:, None] * n
        ai, aj = rc - self.x[i], rc - self.x[j]
        wi, wj = self.w[i], self.w[j]
        vc = self.v[i] + torch.linalg.cross(wi, ai) - self.v[j] - torch.linalg.cross(wj, aj)
        th1 = torch.linalg.cross(B["n"], n)
        th2 = _dot(0.5 * (wi + wj) * dt, n)[:, None] * n
        Fs = self._turn(self._turn(B["Fs"], th1), th2)
        Tb = self._turn(self._turn(B["Tb"], th1), th2)
        Rb = gamma * torch.minimum(self.r[i], self.r[j])
        A, I = Rb * Rb * math.pi, Rb ** 4 / 4.0 * math.pi
        kn = Eb / (self.r[i] + self.r[j])
        ks = kn / knks
        dn = _dot(vc, n)[:, None] * n * dt
        wr = wi - wj
        rn = _dot(wr, n)[:, None] * n * dt
        Fn = B["Fn"] - _dot(dn, n) * kn * A
        Fs = Fs - (vc * dt - dn) * (ks * A)[:, None]
        Tt = B["Tt"] - _dot(rn, n) * ks * 2.0 * I
        Tb = Tb - (wr * dt - rn) * (kn * I)[:, None]
        smax = -Fn / A + Tb.norm(dim=1) / I * Rb
        tmax = Fs.norm(dim=1) / A + Tt.abs() / (2.0 * I) * Rb
        broke = torch.zeros_like(was)
        if sigma > 0:
            broke |= smax > sigma
        if C > 0:
            broke |= tmax > C - mu * smax
        w1, w3 = was, was[:, None]
        Fn, Tt = torch.where(w1, Fn, 0.0 * Fn), torch.where(w1, Tt, 0.0 * Tt)
        Fs, Tb = torch.where(w3, Fs, 0.0 * Fs), torch.where(w3, Tb, 0.0 * Tb)
        self.bonds = {"b": B["b"], "n": torch.where(w3, n, B["n"]), "Fs": Fs, "Tb": Tb, "Fn": Fn, "Tt": Tt,
                      "ok": was & ~broke}
        f = Fn[:, None] * n + Fs
        t = Tt[:, None] * n + Tb
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        T.index_add_(0, i, t + torch.linalg.cross(ai, f))
        T.index_add_(0, j, -t - torch.linalg.cross(aj, f))

    def forces(self, dt, wall_dt):
        F, T = torch.zeros_like(self.x), torch.zeros_like(self.x)
        self._contacts(F, T, dt)
        if self.bonds is not None:
            self._bonded(F, T, dt)
        if self.tri is not None:
            self._plane(F, T, wall_dt)
        if self.k and self.fc is not None:
            F += self.fc
        if self.k and self.extra is not None:
            F += self.extra[0]
            T += self.extra[1]
        self.F, self.T = F, T

    def _kick(self, drift):
        h = 0.5 * self.dt
        if self.nc:
            c = self.cl[self.peb]
            f = self.F[self.peb]
            Fc = torch.zeros_like(self.cx).index_add_(0, c, f)
            arm = self.x[self.peb] - self.cx[c]
            Tc = torch.zeros_like(self.cx).index_add_(0, c, self.T[self.peb] + torch.linalg.cross(arm, f))
            q0, q = self.cq[:, 0], self.cq[:, 1:]
            u = torch.zeros(self.nc, 3, 3, dtype=torch.float64, device=q.device)
            u[:, 0, 1], u[:, 0, 2], u[:, 1, 0] = -q[:, 2], q[:, 1], q[:, 2]
            u[:, 1, 2], u[:, 2, 0], u[:, 2, 1] = -q[:, 0], -q[:, 1], q[:, 0]
            R = torch.eye(3, dtype=torch.float64, device=q.device) + 2.0 * q0[:, None, None] * u + 2.0 * (u @ u)
            self.cv = self.cv + (Fc * self.cim[:, None] + self.g) * h
            self.cw = self.cw + (R @ self.cI @ R.transpose(1, 2) @ Tc[..., None])[..., 0] * h
            if drift:
                self.cx = self.cx + self.dt * self.cv
                s = 0.5 * self.dt * self.cw
                dq0 = -_dot(q, s)
                dq = q0[:, None] * s + torch.linalg.cross(s, q)
                cq = torch.cat([(q0 + dq0)[:, None], q + dq], 1)
                self.cq = cq / cq.norm(dim=1, keepdim=True)
            self.w[self.peb] = self.cw[c]
            self.v[self.peb] = self.cv[c] + torch.linalg.cross(self.cw[c], self.x[self.peb] - self.cx[c])
        free = ((self.cl < 0) & (self.im > 0))[:, None]
        self.v = torch.where(free, self.v + (self.F * self.im[:, None] + self.g) * h, self.v)
        I = 0.4 * self.r ** 2 / torch.where(self.im > 0, self.im, torch.ones_like(self.im))
        self.w = torch.where(free, self.w + self.T / I[:, None] * h, self.w)
        if drift:
            self.x = self.x + self.dt * self.v

    def step(self):
        self.k += 1
        self.forces(0.5 * self.dt, self.dt)
        self._kick(True)
        self.forces(0.5 * self.dt, self.dt)
        self._kick(False)

    def out(self):
        got = {"position": self.x, "velocity": self.v, "angularVelocity": self.w, "force": self.F, "torque": self.T}
        return {k: v.cpu().numpy() for k, v in got.items()}


# ---------------------------------------------------------- exact: coupling --
def _marker_offsets(R, dx, h):
    """Shells of golden-angle points inside a ball's surface."""
    out = []
    layer = 0
    while layer * dx < 2.0 * h and R - (layer + 0.5) * dx > 0.25 * dx:
        r = R - (layer + 0.5) * dx
        n = max(1, int(math.floor(4.0 * math.pi * r * r / (dx * dx) + 0.5)))
        k = np.arange(n)
        z = 1.0 - (2.0 * k + 1.0) / n
        s, phi = np.sqrt(np.maximum(0.0, 1.0 - z * z)), math.pi * (3.0 - math.sqrt(5.0)) * k
        out.append(r * np.stack([s * np.cos(phi), s * np.sin(phi), z], 1))
        layer += 1
    return np.concatenate(out) if out else np.zeros((1, 3))


def _exact_coupled(case, seed):
    sc = _coupled_scene(case, seed)
    fluid, balls = _Fluid(sc.sph), _Balls(sc.dem)
    offs = [_marker_offsets(R, sc.marker_spacing, sc.marker_h) for R in sc.dem.radius]
    of = torch.as_tensor(np.repeat(np.arange(len(offs)), [len(o) for o in offs]), device=balls.x.device)
    off = _t(np.concatenate(offs))
    l = off.norm(dim=1, keepdim=True)
    normal = torch.where(l > 0, off / l.clamp(min=1e-300), torch.zeros_like(off))
    fluid.bounds.append([None, None, normal])
    for _ in range(WARM + case["steps"]):
        fluid.bounds[1][0] = balls.x[of] + off
        fluid.bounds[1][1] = balls.v[of] + torch.linalg.cross(balls.w[of], off)
        re = torch.zeros_like(off)
        fluid.step(re)
        re *= 0.5
        force = torch.zeros_like(balls.x).index_add_(0, of, re)
        torque = torch.zeros_like(balls.x).index_add_(0, of, torch.linalg.cross(off, re))
        balls.extra = (force, torque)
        balls.step()
        balls.step()
    return {"fluid": fluid.out(), "balls": balls.out(), "force": force.cpu().numpy(), "torque": torque.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "coupled":
        return _exact_coupled(case, seed)
    if case["kind"] == "sph":
        f = _Fluid(_sph_scene(case, seed))
        for _ in range(WARM + case["steps"]):
            f.step()
        return f.out()
    if case["kind"] == "batch":
        got = []
        for sc in _batch_scenes(case, seed):
            f = _Fluid(sc)
            for _ in range(WARM + case["steps"]):
                f.step()
            got.append(f.out(("position", "velocity", "density", "pressure", "densityChange")))
        return got
    d = _Balls(_dem_scene(case, seed))
    for _ in range(WARM + case["steps"]):
        d.step()
    out = {"balls": d.out()}
    if case["kind"] == "beam":
        q = d.cq.cpu().numpy()
        out["clumps"] = {"position": d.cx.cpu().numpy(), "velocity": d.cv.cpu().numpy(),
                         "angularVelocity": d.cw.cpu().numpy(), "orientation": q}
        b = d.bonds
        # bonds in the library's order are not these: compared are the balls' sums
        out["bonds"] = {"isBonded": None, "normalForce": None, "shearForce": None, "bendingTorque": None}
    return out
