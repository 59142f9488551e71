"""Performance cases of the GB300 dual-particle SPH liquid, the DEM sand and the
warm-start training, each run through the public entry points.

A liquid pass is what a program does with a scene: the particle state goes in
(host FP64, pinned), ``initialize``, a number of ``advance`` steps (a frame's
worth or part of one), and the state comes back to the host, where it becomes
the FP32 positions and velocities of a frame.  Every pass starts from the same
state, so its work does not depend on how many passes ran before.  A sand pass
is the same without ``initialize`` (a loaded frame goes on with the boundary
that was set up once).  Particles and velocities are the library's FP32 (liquid)
or float-float / FP32 (sand) state, handed out as FP64.

``exact`` restates each path in 64 bits with torch alone.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sand-water-coupling_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import swc  # noqa: E402
from swc import learn, scenes  # noqa: E402

MODEL = os.path.join(PKG, "swc", "models", "warm_start.npz")
GATE = 2  # learned start: the gate that the benchmark uses
DP = C.POINTER(C.c_double)


def listed():
    return [
        # the smallest liquid anyone runs: the 2D dam break (3,200 particles) with the
        # reference's own warm start, one frame of 1/60 s at dt = 1e-3
        {"name": "dam_break_2d", "kind": "liquid", "scene": "dam2", "nx": 40, "ny": 80, "start": "prefix", "steps": 17},
        # a finer 2D tank, odd size, previous pressure of the same node
        {"name": "block_2d_n295", "kind": "liquid", "scene": "block2", "n": 295, "start": "node", "steps": 12},
        # a preview-sized 3D block, one frame of 1/60 s at dt = 5e-4
        {"name": "block_3d_n25", "kind": "liquid", "scene": "block3", "n": 25, "start": "extrapolate", "steps": 33},
        # a ragged 3D column with free surfaces and the reference's warm start
        {"name": "column_3d_77x53x41", "kind": "liquid", "scene": "dam3", "nx": 77, "ny": 53, "nz": 41,
         "start": "prefix", "steps": 8},
        # the 3D dam break (524,288 particles), half a frame
        {"name": "dam_break_3d", "kind": "liquid", "scene": "dam3", "nx": 128, "ny": 64, "nz": 64,
         "start": "extrapolate", "steps": 16},
        # the benchmark block (2,097,152 particles) with the shipped network and the gate
        {"name": "block_3d_n128", "kind": "liquid", "scene": "block3", "n": 128, "start": "learned", "steps": 16},
        # a tank of 3M particles with a turning paddle of 250k boundary particles
        {"name": "paddle_tank_3m", "kind": "liquid", "scene": "tank", "n": 3_000_000, "start": "extrapolate", "steps": 4},
        # the projection alone (VirtualParticle::project), with the virtual particles read back
        {"name": "project_3d_n64", "kind": "project", "scene": "block3", "n": 64, "start": "zero"},
        # the sand demo at its own size (247 particles in 2D), calls of a few microseconds
        {"name": "sand_2d_s30", "kind": "sand", "dim": 2, "scale": 30, "steps": 17},
        # a mid-sized 3D heap (39,754 particles)
        {"name": "sand_3d_s60", "kind": "sand", "dim": 3, "scale": 60, "steps": 17},
        # the benchmark's sand block (2,009,840 particles)
        {"name": "sand_3d_s225", "kind": "sand", "dim": 3, "scale": 225, "steps": 8},
        # one epoch of the warm-start network's training at the recipe's batch size
        {"name": "train_epoch_200k", "kind": "train", "rows": 200_003, "batch": 4096},
    ]


def fitting(cells, brick, nodes=lambda n: n + 7):
    """The next size from `cells` on whose node lattice leaves at most four nodes of its last
    brick along x empty.  With more, the virtual gather of the code that these cases were
    first measured on reads past its cell ranges where liquid fills the lattice's last corner."""
    while -nodes(cells) % brick > 4:
        cells += 1
    return cells


def tank_cells(c):
    """Cells along an axis of the dam break's domain, one and a half times the column."""
    return int(round(round(0.015 * c, 2) / 0.01))


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    start = rng.choice(["prefix", "node", "zero", "extrapolate", "learned"])
    kind = rng.choice(["dam2", "block2", "block3", "dam3", "block3", "dam3", "tank", "project", "sand2", "sand3",
                       "sand3", "train"])
    if kind == "dam2":
        return {"kind": "liquid", "scene": "dam2", "nx": size(11, 80), "ny": size(11, 80), "start": start,
                "steps": rng.randint(3, 17)}
    if kind == "block2":
        return {"kind": "liquid", "scene": "block2", "n": fitting(size(24, 420), 16), "start": start, "steps": rng.randint(3, 12)}
    if kind == "block3":
        return {"kind": "liquid", "scene": "block3", "n": fitting(size(9, 110), 8), "start": start, "steps": rng.randint(3, 10)}
    if kind == "dam3":
        return {"kind": "liquid", "scene": "dam3", "nx": fitting(size(15, 150), 8, lambda n: tank_cells(n) + 7),
                "ny": size(11, 90), "nz": size(11, 80), "start": start, "steps": rng.randint(3, 10)}
    if kind == "tank":
        return {"kind": "liquid", "scene": "tank", "n": size(100_000, 2_500_000), "start": start,
                "steps": rng.randint(2, 4)}
    if kind == "project":
        return {"kind": "project", "scene": "block3", "n": fitting(size(10, 90), 8), "start": rng.choice(["zero", "prefix"])}
    if kind == "sand2":
        return {"kind": "sand", "dim": 2, "scale": size(12, 300), "steps": rng.randint(3, 17)}
    if kind == "sand3":
        return {"kind": "sand", "dim": 3, "scale": size(12, 200), "steps": rng.randint(3, 12)}
    return {"kind": "train", "rows": size(2_000, 400_000), "batch": rng.choice([1024, 4096, 16384])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def liquid_scene(case, seed):
    kind = case["scene"]
    if kind == "dam2":
        s = scenes.dam_break_2d(seed=seed, width_cells=case["nx"], height_cells=case["ny"])
    elif kind == "block2":
        s = scenes.projection_block_2d(n=case["n"], seed=seed)
    elif kind == "block3":
        s = scenes.projection_block_3d(n=case["n"], seed=seed)
    elif kind == "dam3":
        cells = (case["nx"], case["ny"], case["nz"])
        s = scenes.dam_break_3d(seed=seed, cells=cells, domain=tuple(round(0.015 * c, 2) for c in cells))
    else:
        # tank of 256 x 128 x 128 lattice cells, filled from the floor, an upright blade in it
        s = scenes.paddle_tank_3d(seed=seed, n_fluid=case["n"], domain=(2.56, 1.28, 1.28), paddle_particles=250_000,
                                  paddle_half=(0.05, 0.35, 0.2))
    return s.rounded_to_float32()


def sand_scene(case, seed):
    """The builder's packed block (half-length 1/8, every touching pair overlapping by
    1e-4) in the corner of a container of half-length 1/6, walls 8r deep."""
    dim, r = case["dim"], 1.0 / (4 * case["scale"])
    rng = np.random.default_rng(seed)
    half, wall = 0.125, 1.0 / 6
    x = scenes.packed_box(dim, r, np.zeros(dim), np.ones(dim) * half) * 0.9999
    lo = x.min(axis=0)
    x[:, :2] += (-wall + 1.5 * r - lo)[:2]
    v = rng.normal(0.0, 0.01, x.shape).astype(np.float32).astype(np.float64)
    bx, bn = scenes.complement_box_boundary(dim, r, -wall * np.ones(dim), wall * np.ones(dim), np.zeros(dim),
                                            np.ones(dim) * (wall + 10 * r), depth=8 * r)
    return scenes.SandScene(name="sand", dim=dim, radius=r, mass=1000.0 / x.shape[0], positions=x, velocities=v,
                            boundary_positions=bx, boundary_normals=bn.astype(np.float32).astype(np.float64))


def train_rows(case, seed):
    g = torch.Generator().manual_seed(seed)
    f = torch.randn(case["rows"], learn.N_IN, generator=g)
    f = f * torch.linspace(0.5, 2.0, learn.N_IN) + torch.linspace(-1.0, 1.0, learn.N_IN)
    t = torch.sin(f[:, 3]) + 0.5 * f[:, 4] * f[:, 0] + 0.1 * torch.randn(case["rows"], generator=g)
    return f.numpy(), t.numpy()


def pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64))
    return t.pin_memory() if torch.cuda.is_available() else t


class State:
    pass


def prepare(case, seed):
    s = State()
    s.kind = case["kind"]
    if s.kind == "train":
        f, t = train_rows(case, seed)
        s.norm, s.params = learn.normalisation(f, t), learn.init_params(seed)
        s.trainer = learn.Trainer(f.shape[0], case["batch"])
        s.trainer.add(f, t)
        return s
    if s.kind == "sand":
        sc = sand_scene(case, seed)
        s.sim = swc.DEMParticleSand.from_scene(sc)
        s.sim.initialize()
        s.get = s.sim.L.swc_sand_get_particles
    else:
        sc = liquid_scene(case, seed)
        s.sim = swc.DualParticleSphLiquid(sc, warm_start=case["start"], learned_gate=GATE,
                                          keep_virtual_velocity=s.kind == "project")
        if case["start"] == "learned":
            s.sim.setMlp(*learn.load_model(MODEL))
        s.sim.initialize()
        s.get = s.sim.L.swc_get_particles
    s.dt, s.steps, s.n = sc.dt, case.get("steps", 1), sc.n_particles
    s.x, s.v = pinned(sc.positions), pinned(sc.velocities)
    s.ox, s.ov = torch.empty_like(s.x, pin_memory=s.x.is_pinned()), torch.empty_like(s.x, pin_memory=s.x.is_pinned())
    s.fx, s.fv = torch.empty(s.x.shape, dtype=torch.float32), torch.empty(s.x.shape, dtype=torch.float32)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def read_back(s):
    rc = s.get(s.sim.h, C.cast(s.ox.data_ptr(), DP), C.cast(s.ov.data_ptr(), DP), s.n)
    if rc:
        raise swc.SwcError(rc, "get_particles")
    s.fv.copy_(s.ov)


def run(s):
    if s.kind == "train":
        s.trainer.set_params(s.params, s.norm)
        loss = s.trainer.fit(epochs=1, lr=1e-3, seed=7)
        return {"params": s.trainer.params()[0], "loss": loss}
    s.sim.setParticles(s.x.numpy(), s.v.numpy())
    if s.kind == "sand":
        for _ in range(s.steps):
            s.sim.advance(s.dt)
        read_back(s)
        return {"x": s.ox, "v": s.fv}  # float-float positions come back whole in FP64
    if s.kind == "project":
        s.sim.initialize()
        s.sim.project()
        read_back(s)
        v = s.sim.virtual(with_vbar=True)
        out = {k: a.astype(np.float32) for k, a in v.items() if k != "node"}
        return {"node": v["node"], "v": s.fv, **out}
    s.sim.initialize()
    for _ in range(s.steps):
        s.sim.advance(s.dt)
    read_back(s)
    s.fx.copy_(s.ox)
    return {"x": s.fx, "v": s.fv}


# ---------------------------------------------------------------------------
# Work that the path cannot do without
# ---------------------------------------------------------------------------
def counts(case):
    """Particles, boundary particles and lattice nodes within reach, from the sizes alone."""
    kind = case.get("scene")
    if kind == "dam2":
        n, nb, side = case["nx"] * case["ny"], 104**2 - 100**2, (case["nx"] + 3) * (case["ny"] + 3)
    elif kind == "block2":
        n, nb, side = case["n"] ** 2, (case["n"] + 4) ** 2 - case["n"] ** 2, (case["n"] + 5) ** 2
    elif kind == "block3":
        n, nb, side = case["n"] ** 3, (case["n"] + 4) ** 3 - case["n"] ** 3, (case["n"] + 3) ** 3
    elif kind == "dam3":
        c = (case["nx"], case["ny"], case["nz"])
        d = [round(1.5 * k) for k in c]
        n, nb = math.prod(c), math.prod(k + 4 for k in d) - math.prod(d)
        side = math.prod(k + 3 for k in c)
    else:
        n, nb, side = case["n"], 260 * 132 * 132 - 256 * 128 * 128 + 250_000, round(1.1 * case["n"])
    return n, nb, side


def work(case):
    """Bytes: the host arrays in and out and the set-up boundary once, then per step the
    FP32 particle state and the node fields in and out once.  Operations: per step the
    kernel sums over the neighbours within their supports (33 particles and 268 nodes
    in 3D, 13 and 50 in 2D) and the matrix products of CG at its usual count."""
    if case["kind"] == "train":
        macs = 8 * 64 + 64 * 64 + 64
        return {"bytes": 36.0 * case["rows"] * 2, "flops": (6.0 + 2.0) * macs * case["rows"]}
    if case["kind"] == "sand":
        dim, r = case["dim"], 1.0 / (4 * case["scale"])
        n = 0.25**dim / (2 * math.sqrt(3) * r * r if dim == 2 else 4 * math.sqrt(2) * r**3)
        near = 6 if dim == 2 else 12
        return {"bytes": n * (32.0 * dim + case["steps"] * 4 * (6 * dim)), "flops": case["steps"] * n * near * 60.0}
    n, nb, nodes = counts(case)
    dim = 2 if case["scene"] in ("dam2", "block2") else 3
    steps = case.get("steps", 1)
    near, far, stencil = (33, 268, 250) if dim == 3 else (13, 50, 44)
    its = {"prefix": 25, "node": 25, "zero": 38, "extrapolate": 10, "learned": 10}[case["start"]]
    per_step = n * (near * (12 + 25) + far * 18) + nodes * (near * 35 + its * 2 * stencil)
    bytes_ = n * 32.0 * dim + nb * 16.0 + steps * (n * 4 * (2 * dim + 2) * 2 + nodes * 16)
    return {"bytes": bytes_, "flops": float(steps * per_step)}


# ---------------------------------------------------------------------------
# 64-bit restatement
# ---------------------------------------------------------------------------
def spline(h, dim):
    """W(r) and -W'(r)/r of the cubic spline with support h."""
    c0 = (40.0 / 7 / math.pi / h**2) if dim == 2 else (8.0 / math.pi / h**3)
    c1 = 6 * c0 / h

    def w(r):
        q = r / h
        return c0 * torch.where(q < 0.5, 6 * q * q * (q - 1) + 1, 2 * (1 - q).clamp(min=0) ** 3)

    def g(r):
        q = r / h
        inner = c1 * (2 - 3 * q) / h
        return torch.where(q < 0.5, inner, c1 * (1 - q).clamp(min=0) ** 2 / r.clamp(min=1e-300))

    return w, g


class Near:
    """The points of x in cells of side R, and all pairs within R of query points."""

    def __init__(self, x, R):
        self.R, self.dim, self.lo = R, x.shape[1], x.min(0).values
        c = ((x - self.lo) / R).floor().long()
        self.size = c.max(0).values + 1
        order = self.key(c).argsort()
        self.order, self.x = order, x[order]
        n = torch.bincount(self.key(c), minlength=int(self.size.prod()))
        self.start = torch.cat([n.new_zeros(1), n.cumsum(0)])

    def key(self, c):
        k = c[:, -1]
        for a in range(self.dim - 2, -1, -1):
            k = k * self.size[a] + c[:, a]
        return k

    def pairs(self, q, chunk=1 << 19):
        """(query, point, q - x, distance) of all pairs with distance < R, by chunks."""
        shifts = torch.cartesian_prod(*[torch.arange(-1, 2, device=q.device)] * self.dim)
        for b in range(0, q.shape[0], chunk):
            qc = q[b:b + chunk]
            c0 = ((qc - self.lo) / self.R).floor().long()
            for s in shifts:
                c = c0 + s
                inside = ((c >= 0) & (c < self.size)).all(1).nonzero()[:, 0]
                k = self.key(c[inside])
                beg, n = self.start[k], self.start[k + 1] - self.start[k]
                i = inside.repeat_interleave(n)
                j = torch.arange(i.shape[0], device=q.device) + (beg - (n.cumsum(0) - n)).repeat_interleave(n)
                d = qc[i] - self.x[j]
                r = d.square().sum(1).sqrt()
                m = r < self.R
                yield i[m] + b, self.order[j[m]], d[m], r[m]


def exact_liquid(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sc = liquid_scene(case, seed)
    dim, sp = sc.dim, sc.grid_spacing
    T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
    x, v, bx, bn, bv = (T(a) for a in (sc.positions, sc.velocities, sc.boundary_positions, sc.boundary_normals,
                                       sc.boundary_velocities))
    h, H, m = 4 * sc.particle_radius, 4 * sp, sc.mass
    W, G = spline(h, dim)
    WH, GH = spline(H, dim)
    size = list(sc.grid_size[:dim])
    axes = [torch.arange(n, device=dev, dtype=torch.float64) * sp + sc.grid_origin[a] for a, n in enumerate(size)]
    nodes = torch.stack([g.reshape(-1) for g in torch.meshgrid(*axes[::-1], indexing="ij")[::-1]], 1)  # x fastest
    # circular convolution over a lattice padded by the stencil's reach
    off = torch.cartesian_prod(*[torch.arange(-3, 4, device=dev)] * dim)
    off = off[(off.square().sum(1) < 16) & (off.square().sum(1) > 0)]
    r = off.double().square().sum(1).sqrt() * sp
    pad = [n + 4 for n in size[::-1]]
    ker = torch.zeros(pad, dtype=torch.float64, device=dev)
    ker[tuple((off[:, a] % pad[dim - 1 - a]) for a in range(dim - 1, -1, -1))] = -2 * GH(r) * r / (r + 1e-6)
    ker_f = torch.fft.rfftn(ker)
    inner = tuple(slice(0, n) for n in size[::-1])

    def conv(u):
        full = torch.zeros(pad, dtype=torch.float64, device=dev)
        full[inner] = u.view(size[::-1])
        return torch.fft.irfftn(torch.fft.rfftn(full) * ker_f, s=pad)[inner].reshape(-1)

    def density(p, mass):
        rho = p.new_zeros(p.shape[0])
        for i, _, _, r in Near(p, h).pairs(p):
            rho.index_add_(0, i, W(r))
        return mass * rho

    def generate(x, v, rho):
        z = lambda *k: nodes.new_zeros(nodes.shape[0], *k)  # noqa: E731
        wsum, rI, VI, num, den, dvg, gs = z(), z(), z(), z(dim), z(), z(), z(dim)
        for p, u, vol, frac, real in ((x, v, V, m / rho, True), (bx, bv, Vb, Vb, False)):
            for i, j, d, r in Near(p, h).pairs(nodes):
                w, g = W(r), G(r)[:, None] * d
                if real:
                    wsum.index_add_(0, i, w)
                    rI.index_add_(0, i, m * WH(r))
                    VI.index_add_(0, i, vol[j] ** 2 * w)
                num.index_add_(0, i, (frac[j] * w)[:, None] * u[j])
                den.index_add_(0, i, vol[j] * w)
                dvg.index_add_(0, i, vol[j] * (u[j] * g).sum(1))
                gs.index_add_(0, i, vol[j][:, None] * g)
        act = wsum > 1e-6
        vbar = num / (den + 1e-6)[:, None]
        D = dvg - (vbar * gs).sum(1) - kappa * (rI - rho0).clamp(min=0) / rho0
        return act, torch.where(act, VI, 0), rI, vbar, torch.where(act, D, 0)

    def solve(act, VI, D):
        a = -conv(VI)
        a = torch.where(act, a.clamp(min=alpha0), 1)
        # symmetric in u = V p: (a / V) u + C u = D on the active nodes
        diag = torch.where(act, a / VI.where(act, torch.ones_like(VI)), 1)
        op = lambda u: torch.where(act, diag * u + conv(u), 0)  # noqa: E731
        u, res = torch.zeros_like(D), D.clone()
        y = res / diag
        d, ry = y.clone(), res @ y
        for _ in range(4000):
            q = op(d)
            al = ry / (d @ q)
            u += al * d
            res -= al * q
            if res.norm() <= 1e-12 * D.norm():
                break
            y = res / diag
            ry, old = res @ y, ry
            d = y + (ry / old) * d
        return a, u

    rho = density(x, m)
    V, rho0 = m / rho, rho.max()
    Vb = sc.boundary_mass / density(bx, sc.boundary_mass)
    if sc.kappa >= 0:
        kappa = sc.kappa
    else:
        at = lambda k: float(W(torch.tensor(k * sc.particle_radius, dtype=torch.float64)))  # noqa: E731
        kappa = 1 / (at(0) + 6 * at(2) + 6 * at(2 * 3**0.5) if dim == 2 else
                     at(0) + 12 * at(2) + 6 * at(2 * 2**0.5) + 24 * at(2 * 3**0.5))
    act, VI, *_ = generate(x, v, rho)
    alpha0 = float((-conv(VI))[act].max())
    dt, omega = sc.dt, sc.meta.get("paddle_omega", 0.0)
    moving = torch.arange(bx.shape[0], device=dev) >= sc.meta.get("n_walls", bx.shape[0])
    grav = T(sc.gravity[:dim])
    for _ in range(case.get("steps", 1)):
        if case["kind"] == "liquid":
            if omega:
                c, (ca, sa) = T(sc.meta["paddle_center"]), (math.cos(omega * dt), math.sin(omega * dt))
                R = T([[ca, 0, sa], [0, 1, 0], [-sa, 0, ca]])
                bx[moving] = (bx[moving] - c) @ R.T + c
                bn[moving] = bn[moving] @ R.T
                rel = bx[moving] - c
                bv[moving] = torch.stack([omega * rel[:, 2], bv[moving][:, 1], -omega * rel[:, 0]], 1)
            x = x + dt * v
        rho = density(x, m)
        if case["kind"] == "liquid":
            lap = torch.zeros_like(v)
            for i, j, d, r in Near(x, h).pairs(x):
                s = ((v[j] - v[i]) * -d).sum(1) / r.square().clamp(min=1e-300) * G(r) / rho[j]
                lap.index_add_(0, i, s[:, None] * -d)
            v = v + dt * grav + (sc.viscosity * 2 * (dim + 2) * m * dt) * lap
        act, VI, rI, vbar, D = generate(x, v, rho)
        a, u = solve(act, VI, D)
        f = torch.zeros_like(v)
        live = act.nonzero()[:, 0]
        for i, j, d, r in Near(nodes[live], H).pairs(x, 1 << 17):
            f.index_add_(0, i, (u[live][j] * GH(r))[:, None] * d)
        for i, j, d, r in Near(bx, h).pairs(x):
            vn = ((v[i] - bv[j]) * bn[j]).sum(1).clamp(max=0)
            f.index_add_(0, i, -(Vb[j] * vn * W(r))[:, None] * bn[j])
        v = v + f
    if case["kind"] == "project":
        return {"node": live.cpu().numpy(), "v": v, "rho": rI[live], "vol": VI[live], "div": D[live],
                "alpha_hat": a[live], "p": (u[live] / VI[live]), "vbar": vbar[live]}
    return {"x": x, "v": v}


def exact_sand(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sc = sand_scene(case, seed)
    T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
    x, v, bx, bn = (T(a) for a in (sc.positions, sc.velocities, sc.boundary_positions, sc.boundary_normals))
    r0, dt = sc.radius, sc.dt
    Kn, tan = sc.young * r0, math.tan(sc.fric_angle)
    Kt = Kn * sc.poisson
    W, _ = spline(4 * r0, sc.dim)
    near_b = Near(bx, 4 * r0)
    rho = bx.new_zeros(bx.shape[0])
    for i, _, _, r in near_b.pairs(bx):
        rho.index_add_(0, i, W(r))
    Vb = 1 / rho
    norm = lambda a: a.square().sum(1, keepdim=True).sqrt()  # noqa: E731
    for _ in range(case["steps"]):
        x = x + dt * v
        f = torch.zeros_like(v)
        for i, j, d, r in Near(x, 2 * r0).pairs(x):
            n = -d / r.clamp(min=1e-4 * r0)[:, None]  # x_j - x_i over the distance
            w = v[j] - v[i]
            N = Kn * (2 * r0 - r)[:, None] * n
            S = -Kt * (w - (w * n).sum(1, keepdim=True) * n)
            cap = norm(N) * tan
            S = torch.where(norm(S) > cap, S * cap / norm(S).clamp(min=1e-300), S)
            f.index_add_(0, i, torch.where((i != j)[:, None], -(N + S) * dt, 0))
        for i, j, d, r in near_b.pairs(x):
            vn = (v[i] * bn[j]).sum(1, keepdim=True)
            N = -Vb[j][:, None] * vn.clamp(max=0) * bn[j] * W(r)[:, None]
            S = -Kt * (v[i] - vn * bn[j])
            cap, ns = norm(N) * tan, norm(S)
            f.index_add_(0, i, N + torch.where((ns > 1e-6) & ~(cap > ns), S * cap / ns.clamp(min=1e-300), S))
        v = v + f
        v[:, 1] -= 9.8 * dt
    return {"x": x, "v": v}


def exact(case, seed):
    """64-bit values of the outputs; None where they take too long, and for a training
    epoch, whose row order is the library's own."""
    if case["kind"] == "train":
        return None
    if case["kind"] == "sand":
        return exact_sand(case, seed) if case["scale"] <= (300 if case["dim"] == 2 else 110) else None
    return exact_liquid(case, seed) if counts(case)[0] * case.get("steps", 1) <= 3_000_000 else None
