"""The work users have this framework do, as cases to be timed and compared.

Five kinds of call, each through the entry points of a user's program:

  steps    Simulation.step(), ten of them: one period of the sort and collision cadence (nsort = ns_coll = 10)
  solve    Simulation.pdesolver() from the wall potentials, as after a change of the electrode voltages
  window   window_objective() and its backward: gradients of a collisionless FP64 window
  cwindow  collision_window_objective() and its backward: gradients of the collisional mixed-precision window
  dropin   dropin.MainLoop.step(), ten of them: the calls of a Fortran program linked against the library

A case states the cells per axis, the particles per cell and species, whether the argon gas collides with them and
the field and wall voltages.  The plasma is the one of config.py: electrons at 2 eV (5 eV without ions) and Ar+ at
0.026 eV, 1e15 per m^3, cells of 0.1 mm.
"""
import functools
import math

import numpy as np
import torch

from essaitemporaire_lepic_module_b200 import adjoint, config, dropin
from essaitemporaire_lepic_module_b200.sim import Simulation

QE, EPS0, DX = 1.60217646e-19, 8.854187817e-12, 1e-4
BLOBS = 64


def _steps(name, precision, n, ppc, gas, bz, volt, nowait=False):
    return dict(name=name, kind="steps", precision=precision, n1=n[0], n2=n[1], n3=n[2], ppc=ppc, gas=gas, bz=bz,
                volt=volt, ions=True, nowait=nowait)


def listed():
    return [
        # a small box, no field, no gas: 5e5 particles per species, where launches and latencies count
        _steps("steps_mixed_box32", "mixed", (32, 32, 32), 16, False, 0.0, 0.0),
        # an elongated trap between charged end plates in an axial field; no axis a power of two
        _steps("steps_mixed_trap_48x80x112", "mixed", (48, 80, 112), 24, False, 0.02, 20.0),
        # the production run: 1.3e8 particles per species, axial field, argon collisions, no waits in the loop
        _steps("steps_mixed_mcc128", "mixed", (128, 128, 128), 64, True, 0.01, 0.0, True),
        # the FP64 form of a small box, ragged against the 8-cell blocks some kernels use
        _steps("steps_f64_box40x24x32", "f64", (40, 24, 32), 16, False, 0.01, 0.0),
        # the FP64 form at the size it is used for comparisons with the mixed one
        _steps("steps_f64_mcc96", "f64", (96, 96, 96), 32, True, 0.01, 0.0),
        # field solves: a small box, the grid of the production run in FP64, the largest grid with electrodes inside
        dict(name="solve_mixed_48x40x56", kind="solve", precision="mixed", n1=48, n2=40, n3=56, electrodes=False),
        dict(name="solve_f64_128", kind="solve", precision="f64", n1=128, n2=128, n3=128, electrodes=True),
        dict(name="solve_mixed_256", kind="solve", precision="mixed", n1=256, n2=256, n3=256, electrodes=True),
        # gradients of a trap's mean electron energy in the plate voltages, the field and the initial velocities
        dict(name="window_f64_48x48x96", kind="window", n1=48, n2=48, n3=96, ppc=16, bz=0.1, volt=200.0, K=16),
        # gradients of the potential at the centre through collisions
        dict(name="cwindow_mixed_64", kind="cwindow", n1=64, n2=64, n3=64, ppc=32, bz=0.01, volt=0.0, K=12,
             observable="probe"),
        # a Fortran program's loop over arrays in host memory, copied in and out by every call
        dict(name="dropin_16x16x24", kind="dropin", n1=16, n2=16, n3=24, ppc=16, gas=False, bz=0.0, volt=0.0,
             ions=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _axes(rng, cells, step=8, most=160):
    """Three axes, multiples of `step` (the multigrid halves them), of about `cells` cells together."""
    edge = cells ** (1.0 / 3.0)
    r = [rng.uniform(0.7, 1.4) for _ in range(3)]
    return [min(most, max(16, step * int(round(edge * x / step)))) for x in r]


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "solve", "solve", "window", "cwindow", "dropin"])
    if kind == "steps":
        precision = rng.choice(["mixed", "mixed", "f64"])
        n = _axes(rng, _log(rng, 16 ** 3, (112 if precision == "mixed" else 64) ** 3))
        most = 8e7 if precision == "mixed" else 1e7
        ppc = max(2, int(min(_log(rng, 8, 100), most / (n[0] * n[1] * n[2]))))
        gas = rng.random() < 0.3 and n[0] * n[1] * n[2] * ppc > 4e6
        return dict(kind=kind, precision=precision, n1=n[0], n2=n[1], n3=n[2], ppc=ppc, gas=gas,
                    bz=rng.choice([0.0, 0.01, 0.03]), volt=rng.choice([0.0, 5.0, 20.0]), ions=rng.random() < 0.8,
                    nowait=precision == "mixed" and rng.random() < 0.5)
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "f64"])
        n = _axes(rng, _log(rng, 24 ** 3, (176 if precision == "mixed" else 112) ** 3), 16, 224)
        return dict(kind=kind, precision=precision, n1=n[0], n2=n[1], n3=n[2], electrodes=rng.random() < 0.5)
    if kind == "window":
        n = _axes(rng, _log(rng, 16 ** 3, 56 ** 3))
        return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], ppc=rng.randint(4, 16), bz=rng.uniform(0.01, 0.1),
                    volt=rng.choice([20.0, 200.0]), K=rng.randint(6, 16))
    if kind == "cwindow":
        n = _axes(rng, _log(rng, 24 ** 3, 56 ** 3))
        return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], ppc=rng.randint(8, 40), bz=rng.choice([0.01, 0.03]),
                    volt=rng.choice([0.0, 10.0]), K=rng.randint(11, 14), observable=rng.choice(["probe", "energy"]))
    n = _axes(rng, _log(rng, 16 ** 3, 24 ** 3))
    return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], ppc=rng.randint(4, 16), gas=False, bz=rng.choice([0.0, 0.01]),
                volt=rng.choice([0.0, 5.0]), ions=True)


# ---------------------------------------------------------------- set-ups
def _n(c):
    return (int(c["n1"]), int(c["n2"]), int(c["n3"]))


def _levels(n):
    """Multigrid levels: every axis halves down to 3 cells or an odd number."""
    return min((v & -v).bit_length() for v in n)


def _electrodes(n):
    """Two blocks at a third and two thirds of x, a sixteenth of x wide: node ranges (lo, hi), both ends included."""
    e = max(2, n[0] // 16)
    return [[(c - e // 2 + 1, c - e // 2 + 1 + e) for c in (cx, n[1] // 2, n[2] // 2)]
            for cx in (n[0] // 3, 2 * n[0] // 3)]


@functools.lru_cache(maxsize=4)
def _setup(n, ppc, gas, bz, volt, ions, electrodes=False):
    box = [0.0, 0.0, 0.0] + [v * DX * 100.0 for v in n]
    seg, V = [box + [1]], [0.0, 0.0]
    if volt:
        seg += [[0.0, 0.0, 0.0, box[3], box[4], 0.0, -2], [0.0, 0.0, box[5]] + box[3:6] + [-3]]
        V += [volt, volt]
    if electrodes:
        for k, b in enumerate(_electrodes(n)):
            seg.append([(lo - 0.5) * DX * 100.0 for lo, _ in b] + [(hi - 0.5) * DX * 100.0 for _, hi in b] + [-2 - k])
        V += [100.0, -100.0]
    wl = config.Workload("case", n, DX, seg, V, [("[Ar+]", 39.95, 1.0, 0.026, 1.0)] if ions else [],
                         Te=2.0 if ions else 5.0, n0=1e15, ppc=ppc, dt=2e-11 if ions else 1e-11, steps=10,
                         B=(0.0, 0.0, bz), gas_pressure=1.0 if gas else 0.0, ng=_levels(n))
    return config.build(wl)


def _setup_of(c):
    if c["kind"] == "solve":
        return _setup(_n(c), 0, False, 0.0, 0.0, False, bool(c["electrodes"]))
    return _setup(_n(c), int(c["ppc"]), c["kind"] == "cwindow" or bool(c.get("gas")), float(c["bz"]),
                  float(c["volt"]), c["kind"] == "cwindow" or bool(c.get("ions")))


def _cells(c):
    return c["n1"] * c["n2"] * c["n3"]


def _per_species(c):
    return _cells(c) * c["ppc"]


def _particles(c, st, seed):
    """vxp (species, particles, 6): positions uniform in the box, Maxwellian velocities; on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    size = torch.tensor([v * DX for v in _n(c)], dtype=torch.float64, device="cuda")
    out = torch.empty((st.ntype, _per_species(c), 6), dtype=torch.float64, device="cuda")
    for p in range(st.ntype):
        out[p, :, :3] = torch.rand(out.shape[1:2] + (3,), generator=g, dtype=torch.float64, device="cuda") * size
        out[p, :, 3:] = torch.randn(out.shape[1:2] + (3,), generator=g, dtype=torch.float64,
                                    device="cuda") * (st.vt0[p] / math.sqrt(2.0))
    return out


def _on_host(c):
    """Whether the initial particles come from the program's host arrays (else from the GPU loader)."""
    return not c.get("gas") and _per_species(c) <= 1.2e6


def _blobs(c, seed):
    """The source of a field solve: -rho of Gaussian charge blobs, (n3+2, n2+2, n1+2)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n = _n(c)
    at = [torch.tensor(rng.uniform(0, v, BLOBS), device="cuda") for v in n]
    wide = torch.tensor(rng.uniform(2.0, 8.0, BLOBS), device="cuda")
    amp = torch.tensor(rng.uniform(-1e16, 1e16, BLOBS), device="cuda")
    g = [torch.exp(-(torch.arange(-1.0, v + 1.0, dtype=torch.float64, device="cuda")[:, None] - a) ** 2
                   / (2.0 * wide ** 2)) for v, a in zip(n, at)]
    gxy = g[1][:, None, :] * g[0][None, :, :]
    rhs = -QE * torch.matmul(gxy.reshape(-1, BLOBS), (g[2] * amp).t()).t().reshape(n[2] + 2, n[1] + 2, n[0] + 2)
    rhs[0, :, :] = rhs[:, 0, :] = 0.0
    rhs[:, :, 0] = 0.0
    return rhs.contiguous()


def _fixed_order(sim):
    """Every species' particles, sorted by cell, in one order inside each cell."""
    for s in sim.sp:
        n = s.n()
        cell, p = s.cell[:n], s.p[:, :n]
        new = torch.ones_like(cell)
        new[1:] = (cell[1:] != cell[:-1]).to(new.dtype)
        order = torch.argsort(torch.cumsum(new, 0).double() + p[0].double())
        s.cell[:n] = cell[order]
        s.p[:, :n] = p[:, order]


# ---------------------------------------------------------------- the calls
def prepare(c, seed):
    st, kind = _setup_of(c), c["kind"]
    if kind == "steps":
        sim = Simulation(st, precision=c["precision"], nonblocking=bool(c["nowait"]))
        if _on_host(c):
            vxp = _particles(c, st, seed).cpu().numpy()
            sim.load_from_host(vxp, [vxp.shape[1]] * st.ntype)
        else:
            sim.load_uniform(seed=seed + 1)
        return kind, sim
    if kind == "solve":
        sim = Simulation(st, precision=c["precision"])
        sim.rhs.copy_(_blobs(c, seed))
        return kind, sim, sim.phi.clone()
    if kind == "window":
        win = adjoint.Window(st, K=c["K"])
        win.load_uniform(seed=seed + 1)
        V = torch.tensor([0.0, c["volt"], c["volt"]], dtype=torch.float64)
        return kind, win, V, torch.tensor(c["bz"], dtype=torch.float64), win.x0[3:6].clone()
    if kind == "cwindow":
        sim = Simulation(st, precision="mixed")
        sim.load_uniform(seed=seed + 1)
        sim.sort()
        _fixed_order(sim)
        win = adjoint.CollisionWindow(sim, K=c["K"], keep_initial=True, first_it=1)
        V = torch.tensor([0.0] + ([c["volt"]] * 2 if c["volt"] else []), dtype=torch.float64)
        v0 = sim.sp[0].p[3:6, :sim.sp[0].n()].double()
        return kind, win, V, torch.tensor(c["bz"], dtype=torch.float64), v0, c["observable"]
    vxp = _particles(c, st, seed).cpu().numpy()
    room = np.zeros((st.ntype, vxp.shape[1] + 64, 6))
    room[:, :vxp.shape[1]] = vxp
    count = np.full(st.ntype, vxp.shape[1], dtype=np.int32)
    grids = np.zeros((st.ntype,) + st.geom.bcnd.shape)
    dropin.set_commons(st)
    for p in range(st.ntype):
        dropin.charge_deposition(st, room, count, grids, p + 1)
    return kind, dropin.MainLoop(st, room, count, np.zeros(room.shape[:2], dtype=np.int8), grids, collide=False)


def run(state):
    kind, it = state[0], state[1]
    if kind == "steps":
        for _ in range(10):
            it.step()
        return {"phi": it.phi, "E": it.Ei, "density": it.np}
    if kind == "solve":
        it.phi.copy_(state[2])
        it.pdesolver()
        return {"phi": it.phi}
    if kind == "dropin":
        for _ in range(10):
            it.step()
        return {"phi": it.phi, "E": it.Ei, "density": it.np}
    V, Bz, v0 = (t.clone().requires_grad_() for t in state[2:5])
    if kind == "window":
        J = adjoint.window_objective(it, V, Bz, v0)
    else:
        J = adjoint.collision_window_objective(it, V, Bz, v0, observable=state[5])
    J.backward()
    return {"J": J.detach(), "dV": V.grad, "dBz": Bz.grad, "dv0": v0.grad}


# ---------------------------------------------------------------- what a pass needs
def work(c):
    nodes = (c["n1"] + 3) * (c["n2"] + 3) * (c["n3"] + 3)
    kind = c["kind"]
    if kind == "solve":
        # the source and the walls in, phi in and out; a multigrid solve to 1e-10 from zero: about ten cycles of six
        # fine sweeps and a seventh more on the coarser grids, 14 operations a node and sweep
        return {"bytes": nodes * 28.0, "flops": nodes * 10 * 6 * 14 * 8.0 / 7.0}
    if kind in ("steps", "dropin"):
        species = 2 if c["ions"] else 1
        state = 28 if c.get("precision") == "mixed" else 48
        # every step reads and writes each particle; grids: density, phi and E in or out once a step
        per_step = species * _per_species(c) * 2.0 * state + nodes * 8.0 * (2 * species + 2 + 3)
        return {"bytes": 10 * per_step, "flops": 10 * species * _per_species(c) * 200.0}
    if kind == "window":
        # forward: state in and out; backward: state in, adjoint in and out
        return {"bytes": c["K"] * _per_species(c) * 240.0, "flops": c["K"] * _per_species(c) * 700.0}
    return {"bytes": c["K"] * 2 * _per_species(c) * 164.0, "flops": c["K"] * 2 * _per_species(c) * 700.0}


def tolerance(c):
    kind = c["kind"]
    if kind == "solve":
        # phi converged to a residual of 1e-10: FP32 cycles in FP64 refinement end anywhere below 1e-6 of it
        return {"rel": 1e-6, "max": 1e-5} if c["precision"] == "mixed" else {"rel": 1e-8, "max": 1e-7}
    if kind == "steps" and c["gas"]:
        # which particles of a cell collide depends on their order in it, which a counting sort leaves open
        return {"rel": 0.03, "max": 0.9}
    if kind == "steps":
        return {"rel": 1e-5, "max": 4e-4} if c["precision"] == "mixed" else {"rel": 1e-7, "max": 4e-6}
    if kind == "dropin":
        return {"rel": 1e-7, "max": 4e-6}
    # FP64 with field solves to 1e-10; FP32 trajectories and adjoints
    return {"rel": 1e-7, "max": 4e-6} if kind == "window" else {"rel": 5e-5, "max": 5e-3}


# ---------------------------------------------------------------- the same in plain FP64
class _Poisson:
    """A u = b on the plasma nodes 2..n of each axis (fewer where electrodes are), u given on the walls: A is EPS0 times
    the seven-point Laplacian.  Conjugate gradients, preconditioned by the solve of the box without electrodes."""

    def __init__(self, n, plasma, wall):
        self.n, self.plasma, self.wall = n, plasma, wall
        self.S, lam = [], []
        for v in n:
            k = torch.arange(1, v, dtype=torch.float64, device="cuda")
            self.S.append(torch.sin(math.pi / v * k[:, None] * k[None, :]) * math.sqrt(2.0 / v))
            lam.append((2.0 * torch.cos(math.pi * k / v) - 2.0) / DX ** 2)
        self.lam = EPS0 * (lam[2][:, None, None] + lam[1][None, :, None] + lam[0][None, None, :])

    def lap(self, u):
        m = u[1:-1, 1:-1, 1:-1]
        return EPS0 / DX ** 2 * (u[2:, 1:-1, 1:-1] + u[:-2, 1:-1, 1:-1] + u[1:-1, 2:, 1:-1] + u[1:-1, :-2, 1:-1] +
                                 u[1:-1, 1:-1, 2:] + u[1:-1, 1:-1, :-2] - 6.0 * m)

    def box(self, r):
        sx, sy, sz = self.S

        def sines(a):
            a = torch.matmul(a, sx)
            a = torch.matmul(sy, a)
            return torch.matmul(sz, a.reshape(a.shape[0], -1)).reshape(a.shape)
        return sines(sines(r) / self.lam)

    def solve(self, b):
        """b on the nodes 1..n+1; the result there too, walls included."""
        inside = self.plasma[1:-1, 1:-1, 1:-1]
        u = self.wall.clone()
        r = torch.where(inside, b[1:-1, 1:-1, 1:-1] - self.lap(u), 0.0)
        d, zr_old, size = None, None, float(r.norm())
        x = torch.zeros_like(r)
        full = torch.zeros_like(u)
        for _ in range(200):
            if size == 0.0 or float(r.norm()) <= 1e-14 * size:
                break
            z = torch.where(inside, self.box(r), 0.0)
            zr = (z * r).sum()
            d = z if d is None else z + (zr / zr_old) * d
            zr_old = zr
            full[1:-1, 1:-1, 1:-1] = d
            q = torch.where(inside, self.lap(full), 0.0)
            a = zr / (d * q).sum()
            x += a * d
            r -= a * q
        u[1:-1, 1:-1, 1:-1] += x
        return u


def _walls(c, electrodes=False):
    """On the nodes 1..n+1: which are plasma, and the potential of the others."""
    n = _n(c)
    plasma = torch.zeros((n[2] + 1, n[1] + 1, n[0] + 1), dtype=torch.bool, device="cuda")
    plasma[1:-1, 1:-1, 1:-1] = True
    wall = torch.zeros(plasma.shape, dtype=torch.float64, device="cuda")
    if c.get("volt"):
        wall[0] = wall[-1] = c["volt"]
    if electrodes:
        for b, v in zip(_electrodes(n), (100.0, -100.0)):
            at = tuple(slice(lo - 1, hi) for lo, hi in reversed(b))
            plasma[at] = False
            wall[at] = v
    return plasma, wall


def _in_grid(a, ghost=None):
    """Values on the nodes 1..n+1 inside an array of the nodes 0..n+2, the other nodes from `ghost` (default zero)."""
    full = torch.zeros([v + 2 for v in a.shape], dtype=a.dtype, device=a.device) if ghost is None else ghost.clone()
    full[1:-1, 1:-1, 1:-1] = a
    return full


def _ghosts(c):
    """The potential of the walls, ghost planes included."""
    g = torch.zeros((c["n3"] + 3, c["n2"] + 3, c["n1"] + 3), dtype=torch.float64, device="cuda")
    if c.get("volt"):
        g[:2] = g[-2:] = c["volt"]
    return g


def _field(phi, plasma):
    """E = -grad phi: central differences, and on the walls next to plasma the normal component extrapolated."""
    E = torch.zeros(phi.shape + (3,), dtype=torch.float64, device="cuda")
    diff = torch.zeros_like(E)
    for a, axis in enumerate((2, 1, 0)):
        diff[..., a] = -(torch.roll(phi, -1, axis) - torch.roll(phi, 1, axis)) / (2.0 * DX)
    E = torch.where(plasma[..., None], diff, E)
    out = E.clone()
    core = torch.zeros_like(plasma)
    core[1:-1, 1:-1, 1:-1] = True
    for a, axis in enumerate((2, 1, 0)):
        for way in (-1, 1):
            there = core & ~plasma & torch.roll(plasma, way, axis)
            far = 2.0 * torch.roll(E, way, axis) - torch.roll(E, 2 * way, axis)
            new = diff.clone()
            new[..., a] = far[..., a]
            out = torch.where(there[..., None], new, out)
    return out


def _exact_steps(c, seed, count):
    st = _setup_of(c)  # only its constants: masses, charges, weights, time step
    n = _n(c)
    plasma, wall = _walls(c)
    poisson = _Poisson(n, plasma, wall)
    ghost = _ghosts(c)
    big = _in_grid(plasma)
    kq = torch.where(big, 1.0, 2.0).double().reshape(-1)
    N1, N2, N3 = n[0] + 3, n[1] + 3, n[2] + 3
    o = torch.tensor([0, 1, 1 + N1, N1], device="cuda")
    o = torch.cat([o, o + N1 * N2])
    parts = [p.clone() for p in _particles(c, st, seed)]

    def spread(x):
        """Base node and the eight weights of the cell around each position."""
        i = torch.floor(x / DX)
        l = 1.0 - (x / DX - i)
        r = 1.0 - l
        i = i.long() + 1
        q = i[:, 0] + N1 * (i[:, 1] + N2 * i[:, 2])
        xy = [l[:, 0] * l[:, 1], r[:, 0] * l[:, 1], r[:, 0] * r[:, 1], l[:, 0] * r[:, 1]]
        return q[:, None] + o, torch.stack([w * l[:, 2] for w in xy] + [w * r[:, 2] for w in xy], 1)

    def deposit(p):
        at, w = spread(parts[p][:, :3])
        g = torch.zeros(N1 * N2 * N3, dtype=torch.float64, device="cuda")
        g.index_add_(0, at.reshape(-1), w.reshape(-1))
        return (g * kq * (st.Nm[p] / DX ** 3)).reshape(N3, N2, N1)

    dens = [deposit(p) for p in range(st.ntype)]
    size = torch.tensor([v * DX for v in n], dtype=torch.float64, device="cuda")
    for _ in range(count):
        rho = sum(float(st.charge[p]) * dens[p] for p in range(st.ntype))
        phi = _in_grid(poisson.solve(-rho[1:-1, 1:-1, 1:-1]), ghost)
        E = _field(phi, big)
        for p in range(st.ntype):
            x, v = parts[p][:, :3], parts[p][:, 3:]
            at, w = spread(x)
            e = (E.reshape(-1, 3)[at] * w[:, :, None]).sum(1)
            k = float(st.dt * st.charge[p] / (2.0 * st.mass[p]))
            v = v + k * e
            if c["bz"]:
                t = torch.tensor([0.0, 0.0, k * c["bz"]], dtype=torch.float64, device="cuda")
                v1 = v + torch.linalg.cross(v, t.expand_as(v))
                v = v + torch.linalg.cross(v1, (2.0 / (1.0 + (k * c["bz"]) ** 2) * t).expand_as(v))
            v = v + k * e
            x = x + st.dt * v
            stays = ((x >= 0) & (x < size)).all(1)
            parts[p] = torch.cat([x, v], 1)[stays]
            dens[p] = deposit(p)
    return {"phi": phi, "E": E, "density": torch.stack(dens)}


def exact(c, seed):
    if c["kind"] == "solve":
        plasma, wall = _walls(c, c["electrodes"])
        u = _Poisson(_n(c), plasma, wall).solve(_blobs(c, seed)[1:, 1:, 1:])
        return {"phi": _in_grid(u)}
    if c["kind"] in ("steps", "dropin") and (c["kind"] == "dropin" or _on_host(c)):
        return _exact_steps(c, seed, 10)
    return None
