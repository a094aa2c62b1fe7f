"""Performance cases of the framework: what its users have it do, through the package's public entry
points (peridem_gb300.sim, peridem_gb300.gen).

A simulation case is a stretch of a run: the handle is made beforehand from a setup, with a
checkpoint of its first state (Sim.snapshot); a pass goes back to the checkpoint (Sim.restore), takes
`steps` explicit steps and reads the node state and the damage, as a driver that saves a frame every
`steps` steps does. Every pass computes the same stretch, so a pass's outputs do not depend on how
often it ran. The geometry of a case (the generator's workloads: shapes, sizes, jittered lattices) is
the case's own, the velocities are the seed's: every particle gets a rigid velocity and a velocity
gradient, so that the bonds of a packing that would be at rest carry elastic waves as they do in a run.
"""
import math
import random

import numpy as np
import torch

from peridem_gb300 import gen
from peridem_gb300.sim import Batch, Sim

MM = 1e-3
SHAPES = 20  # the generator's seed: a case's particles are the same for every seed of prepare()


def listed():
    return [
        # one step and its frame on a few hundred nodes: an interactive probe, all latency
        dict(name="probe_fp32c", kind="impact", precision="fp32c", radius=0.3, steps=1),
        # two-sphere impact at its configured size: contact, breaking, candidate rebuilds; both forms
        dict(name="impact_fp32c", kind="impact", precision="fp32c", radius=1.0, steps=100),
        dict(name="impact_fp64", kind="impact", precision="fp64", radius=1.0, steps=25),
        # 125 rotated cubes in a walled box under gravity
        dict(name="cubes_fp32c", kind="cubes", precision="fp32c", n=5, spacing=0.125, steps=100),
        # touching particles of mixed resolution pressed by a fast wall: contact and fracture
        dict(name="contact_fp32c", kind="contact", precision="fp32c", count=16, steps=40),
        # the crushing packing at its stated parameters (0.9 M nodes, 7.5e7 directed bonds); both forms
        dict(name="crush_fp32c", kind="crush", precision="fp32c", count=512, scale=1.0, steps=50),
        dict(name="crush_fp64", kind="crush", precision="fp64", count=512, scale=1.0, steps=4),
        # the same packing at the size quoted beside it (4.3 M nodes, 4.0e8 directed bonds)
        dict(name="crush_4m_fp32c", kind="crush", precision="fp32c", count=512, scale=0.6, steps=40),
        # one large notched particle hit by a block
        dict(name="plate_fp32c", kind="plate", precision="fp32c", lx=60.0, ly=80.0, steps=50),
        # a server's cohort: independent aggregates in one handle
        dict(name="cohort_fp32c", kind="cohort", precision="fp32c", sims=12, pmin=8, pmax=64, steps=50),
        # a whole small job: the handle from host arrays, a short run, its results, closed again
        dict(name="job_fp32c", kind="job", precision="fp32c", count=32, steps=100),
        # setup generation: the bond lists of 24 particles from their node positions (host to host)
        dict(name="bonds_24", kind="bonds", count=24, scale=0.6),
    ]


def draw(rng: random.Random):
    def spread(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["impact", "impact", "cubes", "contact", "crush", "crush", "plate", "cohort", "job", "bonds"])
    form = rng.choice(["fp32c", "fp32c", "fp64"])
    if kind == "impact":
        return dict(kind=kind, precision=form, radius=round(spread(0.25, 1.5), 3),
                    steps=int(spread(1, 100 if form == "fp32c" else 25)))
    if kind == "cubes":
        return dict(kind=kind, precision=form, n=rng.randint(2, 5), spacing=round(rng.uniform(0.11, 0.2), 4),
                    steps=int(spread(5, 100 if form == "fp32c" else 20)))
    if kind == "contact":
        return dict(kind=kind, precision=form, count=rng.randint(4, 20), steps=int(spread(5, 40 if form == "fp32c" else 8)))
    if kind == "crush":
        scale = round(rng.uniform(0.6, 1.0), 3) if form == "fp32c" else 1.0
        count = int(spread(6, 500 if form == "fp32c" else 400))
        return dict(kind=kind, precision=form, count=count, scale=scale, steps=rng.randint(5, 20) if form == "fp32c" else 3)
    if kind == "plate":
        return dict(kind=kind, precision="fp32c", lx=round(rng.uniform(30, 70), 1), ly=round(rng.uniform(30, 90), 1),
                    steps=rng.randint(5, 30))
    if kind == "cohort":
        return dict(kind=kind, precision="fp32c", sims=rng.randint(2, 14), pmin=rng.randint(4, 16),
                    pmax=rng.randint(17, 64), steps=rng.randint(5, 30))
    if kind == "job":
        return dict(kind=kind, precision=form, count=rng.randint(3, 40), steps=int(spread(10, 100 if form == "fp32c" else 20)))
    return dict(kind="bonds", count=rng.randint(1, 40), scale=round(rng.uniform(0.6, 1.0), 3))


# ---- inputs -----------------------------------------------------------------------------------


def _excite(setup, rng, speed, rate):
    """A rigid velocity of up to `speed` (m/s) and a velocity gradient of up to `rate` (1/s) per particle."""
    for p in range(setup.n_particles):
        s = setup.particle_slice(p)
        x = setup.pos[s]
        setup.vel[s] += rng.uniform(-speed, speed, 3) + (x - x.mean(axis=0)) @ rng.uniform(-rate, rate, (3, 3)).T


def _spacings(scale):
    return tuple(scale * h * MM for h in (0.05, 0.075, 0.1))


def _simulation(case, seed):
    """(setup, config) of a single-simulation case."""
    gen.set_bond_builder("gpu")
    rng = np.random.default_rng((int(seed), 7))
    kind = case["kind"]
    if kind == "impact":
        s, cfg = gen.two_sphere(R=case["radius"] * MM, v=float(rng.uniform(15, 25)), seed=SHAPES)
        _excite(s, rng, 0.5, 500.0)
    elif kind == "cubes":
        s, cfg = gen.cubes125(n=case["n"], h=case["spacing"] * MM, seed=SHAPES)
        _excite(s, rng, 2.0, 500.0)
    elif kind == "contact":
        s, cfg = gen.crush512(box=9.6 * MM, seed=SHAPES, dt=3e-9, hs=_spacings(0.6), count=case["count"])
        cfg.update(wall_z_max=float(s.pos[:, 2].max()) + 0.01 * MM, speed_wall_z_max=-20.0)
        _excite(s, rng, 10.0, 2000.0)
    elif kind == "crush":
        dt = 5e-9 * case["scale"]
        s, cfg = gen.crush512(seed=SHAPES, dt=dt, hs=_spacings(case["scale"]), count=case["count"])
        _excite(s, rng, 2.0, 2000.0)
    elif kind == "plate":
        lx, ly = case["lx"] * MM, case["ly"] * MM
        s, cfg = gen.notched_plate(Lx=lx, Ly=ly, notch_len=0.25 * ly, notch_x=(0.25 * lx, 0.75 * lx), imp_w=0.5 * lx,
                                   v=float(rng.uniform(25, 40)), seed=SHAPES, gap=-0.5)
        _excite(s, rng, 0.5, 50.0)
    else:  # job
        s, cfg = gen.aggregate(case["count"], seed=SHAPES, steps=case["steps"])
        _excite(s, rng, 2.0, 2000.0)
    return s, cfg


def _cohort(case, seed):
    gen.set_bond_builder("gpu")
    rng = np.random.default_rng((int(seed), 11))
    out = []
    for i in range(case["sims"]):
        count = case["pmin"] + (case["pmax"] - case["pmin"]) * i // max(1, case["sims"] - 1)
        s, cfg = gen.aggregate(count, seed=SHAPES + i, steps=2000, wall_speed=float(rng.uniform(0.5, 2.0)))
        _excite(s, rng, 2.0, 2000.0)
        out.append((s, cfg))
    return out


def _points(case, seed):
    """Node positions and bond radii of a packing's particles: the case's shapes, numbered from another node,
    turned and placed by the seed."""
    rng, place = np.random.default_rng(SHAPES), np.random.default_rng((int(seed), 13))
    pos, rad = [], []
    for _ in range(case["count"]):
        kind = ("sphere", "cube", "ellipsoid")[int(rng.integers(3))]
        h = _spacings(case["scale"])[int(rng.integers(3))]
        size = float(rng.uniform(0.6, 1.4)) * MM
        x = gen.lattice(kind, size if kind == "sphere" else size / math.sqrt(3) if kind == "cube" else
                        rng.uniform(0.6, 1.4, 3) * MM, h)
        x = x + rng.uniform(-0.05 * h, 0.05 * h, x.shape)
        x = np.roll(x, int(place.integers(len(x))), axis=0)  # the node numbering starts elsewhere: other pairs
        pos.append(x @ gen.random_rotation(place).T + place.uniform(-6, 6, 3) * MM)
        rad.append(3.0 * h)
    return pos, rad


def prepare(case, seed):
    kind = case["kind"]
    if kind == "bonds":
        return dict(case=case, points=_points(case, seed))
    if kind == "job":
        return dict(case=case, job=_simulation(case, seed))
    if kind == "cohort":
        sims = _cohort(case, seed)
        h = Batch([s for s, _ in sims], [c for _, c in sims], case["precision"])
        h.tune(graphs=1 if h.N < 131072 else -1)  # as the server does: cohorts share the GPU
    else:
        s, cfg = _simulation(case, seed)
        h = Sim(s, cfg, case["precision"])
    h.snapshot()
    return dict(case=case, handle=h)


def run(state):
    case = state["case"]
    if case["kind"] == "bonds":
        return [x.view(np.int32) for x in gen.bonds_gpu(*state["points"])]
    if case["kind"] == "job":
        setup, cfg = state["job"]
        with Sim(setup, cfg, case["precision"]) as h:
            h.step(case["steps"])
            return dict(h.state(), damage=h.damage())
    h = state["handle"]
    h.restore()
    h.step(case["steps"])
    return dict(h.state(), damage=h.damage())


# ---- the work a pass cannot do without ---------------------------------------------------------


def _body(volume, surface, h):
    """(nodes, directed bonds) of a lattice body: 107 partners within 3 h inside, fewer at the surface (a partner at
    distance r is missing with probability r S / 4 V; mean r = 9 h / 4)."""
    n = volume / h ** 3
    return n, n * 107 * max(0.3, 1 - 2.25 * h * surface / (4 * volume))


def _packing(count, scale):
    n = b = 0.0
    for h in _spacings(scale):
        for size in (0.7 * MM, 0.9 * MM, 1.1 * MM, 1.3 * MM):
            ball = _body(math.pi * size ** 3 / 6, math.pi * size ** 2, h)
            e = size / math.sqrt(3)
            cube = _body(e ** 3, 6 * e * e, h)
            n += count / 36 * (2 * ball[0] + cube[0])
            b += count / 36 * (2 * ball[1] + cube[1])
    return n, b


def _size(case):
    kind = case["kind"]
    if kind == "impact":
        r, h = case["radius"] * MM, 0.1 * MM
        n, b = _body(4 / 3 * math.pi * r ** 3, 4 * math.pi * r * r, h)
        return 2 * n, 2 * b
    if kind == "cubes":
        m, h = round(1.0 / case["spacing"]), case["spacing"] * MM
        n, b = _body((m * h) ** 3, 6 * (m * h) ** 2, h)
        return case["n"] ** 3 * n, case["n"] ** 3 * b
    if kind in ("crush", "bonds"):
        return _packing(case["count"], case["scale"])
    if kind == "contact":
        return _packing(case["count"], 0.6)
    if kind == "job":
        return _packing(case["count"], 1.0)
    if kind == "cohort":
        return _packing(case["sims"] * (case["pmin"] + case["pmax"]) / 2, 1.0)
    lx, ly, lz, h = case["lx"] * MM, case["ly"] * MM, 9.0 * MM, 0.5 * MM
    p = _body(lx * ly * lz, 2 * (lx * ly + ly * lz + lx * lz), h)
    q = _body(0.5 * lx * 10 * MM * lz, lx * 10 * MM + 20 * MM * lz + lx * lz, h)
    return p[0] + q[0], p[1] + q[1]


def work(case):
    n, b = _size(case)
    if case["kind"] == "bonds":  # positions in, pairs out; a distance test per directed bond
        return dict(bytes=24 * n + 4 * b, flops=8 * b)
    # a step: 4 B column and 1/8 B live bit per directed bond, 224 B of node state; the frame: 15 doubles and the damage
    w = case["steps"] * (4.125 * b + 224 * n) + 128 * n
    if case["kind"] == "job":  # host arrays in: 17 doubles a node and 8 B a pair
        w += 136 * n + 4 * b
    return dict(bytes=w, flops=case["steps"] * (40 * b + 60 * n))


# ---- the same stretch in 64 bits, plain torch --------------------------------------------------


class _Plain:
    """The explicit step of one simulation (bonds with breaking, self-contact, node contact, walls, external force,
    velocity Verlet) on flat double tensors."""

    CHUNK = 1 << 24

    def __init__(self, s, cfg):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def f(x):
            return torch.as_tensor(np.array(x, dtype=np.float64), device=dev)

        self.s, self.cfg, self.dev = s, cfg, dev
        off = s.node_offset.astype(np.int64)
        cnt = np.diff(off)
        self.pid = torch.as_tensor(np.repeat(np.arange(s.n_particles), cnt), device=dev)
        pairs = s.conn.astype(np.int64) + np.repeat(off[:-1], np.diff(s.conn_offset.astype(np.int64)))[:, None]
        self.i, self.j = (torch.as_tensor(pairs[:, c].copy(), device=dev) for c in (0, 1))
        self.live = torch.ones(len(pairs), dtype=torch.bool, device=dev)
        self.pos, self.disp, self.vel, self.acc, self.ext = (f(x) for x in (s.pos, s.disp, s.vel, s.acc, s.extforce))
        self.vol = f(s.vol)
        self.rho, self.cnot, self.snot = (f(x)[self.pid] for x in (s.rho, s.cnot, s.snot))
        self.breakable = torch.as_tensor(np.asarray(s.breakable) != 0, device=dev)[self.pid]
        self.force = torch.zeros_like(self.pos)
        g = s.geom_wall_info
        self.wall = [float(x) for x in g] if s.allow_wall and g is not None else None
        names = ("x_min", "y_min", "z_min", "x_max", "y_max", "z_max")
        self.speed = [float(cfg.get("speed_wall_" + k, 0.0)) for k in names]
        if self.wall:
            self.wall = [float(cfg.get("wall_" + k, self.wall[c])) for c, k in enumerate(names)]
        self.boxes()

    def boxes(self):
        """Particle boxes as the next step's pair test uses them: those of the positions before its predictor."""
        x, at = self.pos + self.disp, self.pid[:, None].expand(-1, 3)
        z = torch.zeros(self.s.n_particles, 3, dtype=torch.float64, device=self.dev)
        self.lo, self.hi = (z.scatter_reduce(0, at, x, how, include_self=False) for how in ("amin", "amax"))

    def bonds(self):
        f = torch.zeros_like(self.pos)
        for a in range(0, len(self.i), self.CHUNK):
            c = slice(a, a + self.CHUNK)
            i, j, live = self.i[c], self.j[c], self.live[c]
            xi = self.pos[j] - self.pos[i]
            eta = (self.disp[j] - self.disp[i]) + xi
            xn, en = xi.norm(dim=1), eta.norm(dim=1)
            st = (en - xn) / xn
            t = (self.cnot[i] * st / en * live)[:, None] * eta
            f.index_add_(0, i, t * self.vol[j][:, None])
            f.index_add_(0, j, t * -self.vol[i][:, None])
            self.live[c] = live & ~(self.breakable[i] & (st > self.snot[i]))
        return f

    def close(self):
        """Node pairs (i < j) within the contact radius: one pass over cells of that edge and their neighbours."""
        x = self.pos + self.disp
        cell = torch.floor((x - x.amin(0)) / (self.s.contact_radius * (1 + 1e-9))).long() + 1
        dim = cell.amax(0) + 2
        key = (cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2]
        key, at = torch.sort(key)
        got = []
        for d in range(14):  # the cell itself and 13 of its neighbours: each pair of cells once
            dx, dy, dz = (d + 13) // 9 - 1, (d + 13) // 3 % 3 - 1, (d + 13) % 3 - 1
            to = key + (dx * dim[1] + dy) * dim[2] + dz
            lo, hi = torch.searchsorted(key, to), torch.searchsorted(key, to, right=True)
            if d == 0:
                lo = torch.arange(1, len(key) + 1, device=self.dev)
            n = (hi - lo).clamp(min=0)
            a = torch.repeat_interleave(torch.arange(len(key), device=self.dev), n)
            b = torch.arange(len(a), device=self.dev) - torch.repeat_interleave(n.cumsum(0) - n, n) + lo[a]
            i, j = at[a], at[b]
            near = (x[j] - x[i]).square().sum(1) <= self.s.contact_radius ** 2
            got.append(torch.stack([torch.minimum(i, j)[near], torch.maximum(i, j)[near]]))
        return torch.cat(got, 1)

    def pair(self, i, j, ref, stiff):
        """Normal, damping and friction force densities on i from j (with j's volume, i's density)."""
        s = self.s
        d = (self.pos[j] + self.disp[j]) - (self.pos[i] + self.disp[i])
        dn = d.norm(dim=1)
        u = d / dn[:, None]
        fc = (stiff * (dn - ref) / ref * self.vol[j])[:, None] * u
        rel = self.vel[i] - self.vel[j]
        rn = (rel * u).sum(1)
        fd = (-2 * s.damping_ratio * torch.sqrt(stiff * self.rho[i]) * torch.sqrt(self.vol[j]) * rn)[:, None] * u
        rt = rel - rn[:, None] * u
        v = rt.norm(dim=1)
        mag = s.friction_coefficient * fc.norm(dim=1)
        mag = torch.where(v < mag * self.cfg["dt"] / self.rho[i], v / self.rho[i] / self.cfg["dt"], mag)
        ff = torch.where((v > 0)[:, None], rt * (-mag / v.clamp(min=1e-300))[:, None], torch.zeros_like(rt))
        return dn, fc, fd, ff

    def contact(self, f):
        s = self.s
        i, j = self.close()
        if not len(i):
            return
        rc, stiff = s.contact_radius, s.normal_stiffness * s.contact_radius
        own = self.pid[i] == self.pid[j]
        p, q = self.pid[i], self.pid[j]
        meet = ((self.lo[p] - rc <= self.hi[q]) & (self.hi[p] + rc >= self.lo[q])).all(1)
        a, b = i[~own & meet], j[~own & meet]
        if len(a):
            dn, fc, fd, ff = self.pair(a, b, torch.full_like(self.vol[a], rc), torch.full_like(self.vol[a], stiff))
            on = (dn < rc)[:, None]
            f.index_add_(0, a, (fc + fd + ff) * on)
            r = (self.vol[a] / self.vol[b])[:, None]
            f.index_add_(0, b, -(fc * r + fd * torch.sqrt(r) + ff) * on)
        a, b = i[own], j[own]
        if len(a):
            key = self.i * len(self.pos) + self.j  # ascending: the setup's lists are sorted
            k = torch.searchsorted(key, a * len(self.pos) + b).clamp(max=len(key) - 1)
            free = ~((key[k] == a * len(self.pos) + b) & self.live[k])
            a, b = a[free], b[free]
            for p, q in ((a, b), (b, a)):
                xn = (self.pos[q] - self.pos[p]).norm(dim=1)
                short = xn < rc
                ref = torch.where(short, xn, torch.full_like(xn, rc))
                dn, fc, fd, ff = self.pair(p, q, ref, torch.where(short, self.cnot[p], torch.full_like(xn, stiff)))
                f.index_add_(0, p, (fc + fd + ff) * ((dn < ref) & self.breakable[p])[:, None])

    def walls(self, f):
        s, R, mu = self.s, self.s.contact_radius, self.s.friction_coefficient
        x = self.pos + self.disp
        for face in range(6):
            c = face % 3
            dist = x[:, c] - self.wall[face]
            n = torch.nonzero(dist.abs() <= R)[:, 0]
            if not len(n):
                continue
            sign, d = torch.where(dist[n] > 0, 1.0, -1.0).double(), dist[n].abs()
            area = math.pi / 3 * (R - d) ** 2 * (2 * R - d)
            depth = (R - math.pi / 4 * (R * R - d * d) ** 2 / area).clamp(min=0)
            F = s.normal_stiffness * depth * area
            rel = self.vel[n].clone()
            rel[:, c] -= self.speed[face]
            t = rel.clone()
            t[:, c] = 0
            v = t.norm(dim=1)
            mag = torch.where(v < mu * F * self.cfg["dt"] / self.rho[n], v / self.rho[n] / self.cfg["dt"], mu * F)
            add = torch.where((v > 0)[:, None], t * (-mag / v.clamp(min=1e-300))[:, None], torch.zeros_like(t))
            add[:, c] = sign * F - 2 * s.damping_ratio * torch.sqrt(s.normal_stiffness * self.rho[n]) * torch.sqrt(area) * rel[:, c]
            f.index_add_(0, n, add)

    def step(self):
        dt = self.cfg["dt"]
        self.disp = self.disp + dt * self.vel + 0.5 * dt * dt * self.acc
        f = self.bonds()
        if self.wall:
            self.walls(f)
        f += self.ext
        self.contact(f)
        an = f / self.rho[:, None]
        self.vel = self.vel + 0.5 * dt * (self.acc + an)
        self.acc, self.force = an, f
        self.boxes()
        if self.wall:
            self.wall = [w + v * dt for w, v in zip(self.wall, self.speed)]

    def state(self):
        n = len(self.pos)
        ends = torch.cat([self.i, self.j])
        was = torch.bincount(ends, minlength=n).double()
        now = torch.bincount(ends[torch.cat([self.live, self.live])], minlength=n).double()
        return dict(curpos=self.pos + self.disp, vel=self.vel, acc=self.acc, force=self.force, disp=self.disp,
                    damage=(was - now) / was)


def exact(case, seed):
    if case["kind"] == "bonds":
        return None  # whole numbers
    sims = _cohort(case, seed) if case["kind"] == "cohort" else [_simulation(case, seed)]
    got = []
    for s, cfg in sims:
        p = _Plain(s, cfg)
        for _ in range(case["steps"]):
            p.step()
        got.append(p.state())
        del p
    return {k: torch.cat([g[k] for g in got]).cpu().numpy() for k in got[0]}
