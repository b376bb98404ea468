"""The work that programs using this library have it do, as timed cases.

Four kinds of pass, each through the public entry points (sca2012_b200.Solver
and the C-ABI it wraps):

  frame    one SPHSystem::animation() of the reference's own units and rules:
           records up, one adaptive step, records down (and, in display mode
           2, the surface mesh): what a program that moved over from the
           reference does per frame.
  run      an SI-unit simulation from given particles: records up, K steps,
           records down (and the surface mesh of the last surface step).
  batch    many walled scenes advanced together: state up, K steps, records
           down.
  rollout  one iteration of a fit through the differentiable rollout: state
           up, checkpointed forward, density-grid loss, backward; the loss,
           the grid and every gradient come back.

Every pass starts from the particles its state holds, so a pass can be
repeated and gives the same outputs each time.  Fluids are jittered lattice
blocks in the low corner of their box (the repository's own scenes), with
velocities drawn N(0, 0.1^2) m/s as the differentiable workload draws them.
"""
import ctypes
import math

import numpy as np
import torch

import sca2012_b200 as sph
from sca2012_b200 import scenes

REST = 1000.0      # SI rest density
GRAVITY = -9.8
GRID_LOSS = 32     # nodes per axis of the rollout's loss grid


def _case(name, kind, **kw):
    return dict(name=name, kind=kind, **kw)


def listed():
    return [
        # the reference's three apps at their own starting sizes, split and
        # merge on, one frame per pass: launches and latency
        _case("frame_2d", "frame", solver="2d", nx=32, ny=63, nz=1, surface=False),
        _case("frame_3d2_surface", "frame", solver="3d2", nx=19, ny=20, nz=19, surface=True),
        _case("frame_3d4", "frame", solver="3d4", nx=94, ny=11, nz=46, surface=False),
        # the 4,096-particle 2D dam, stepped by persistent launches
        _case("dam_2d_4k", "run", dim=2, spacing=0.01, nx=64, ny=64, nz=1, ways=2, adaptive=False, steps=100,
              mode="persistent", jitter=0.01, surface=False),
        # an ordinary plain 3D block of odd sizes, replayed as graphs
        _case("plain_3d_ragged", "run", dim=3, spacing=0.01, nx=61, ny=47, nz=33, ways=2, adaptive=False, steps=20,
              mode="graph", jitter=0.1, surface=False),
        # the 131,072-particle two-way adaptive dam, past the 50 steps after which split groups merge back
        _case("adaptive_3d_131k", "run", dim=3, spacing=0.01, nx=64, ny=64, nz=32, ways=2, adaptive=True, steps=60,
              mode="launches", jitter=0.01, surface=False),
        # a million particles: plain, and four-way adaptive with the surface every 10 steps
        _case("plain_3d_1m", "run", dim=3, spacing=0.005, nx=128, ny=128, nz=64, ways=4, adaptive=False, steps=10,
              mode="launches", jitter=0.05, surface=False),
        _case("adaptive_3d_1m_surface", "run", dim=3, spacing=0.005, nx=128, ny=128, nz=64, ways=4, adaptive=True,
              steps=20, mode="launches", jitter=0.01, surface=True),
        # batches of independent dam breaks
        _case("batch_2d", "batch", dim=2, spacing=0.01, scenes=48, n_min=1024, n_max=16384, ways=2, steps=100),
        _case("batch_3d", "batch", dim=3, spacing=0.01, scenes=24, n_min=1024, n_max=32768, ways=2, steps=100),
        # fits through the rollout: a small plain block, and the 32^3 adaptive one
        _case("rollout_3d_4k", "rollout", dim=3, spacing=0.01, nx=16, ny=16, nz=16, adaptive=False, steps=20, every=10),
        _case("rollout_3d_32k", "rollout", dim=3, spacing=0.01, nx=32, ny=32, nz=32, adaptive=True, steps=60, every=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, n, dim):
    """Counts per axis of about n particles, each axis off the cube by up to 1.6."""
    side = n ** (1.0 / dim)
    f = [math.exp(rng.uniform(-0.47, 0.47)) for _ in range(dim)]
    g = math.prod(f) ** (1.0 / dim)
    c = [max(4, int(round(side * v / g))) for v in f]
    return c + [1] * (3 - dim)


def draw(rng):
    kind = rng.choice(["frame", "run", "run", "run", "batch", "rollout"])
    if kind == "frame":
        solver = rng.choice(["2d", "3d2", "3d4"])
        if solver == "2d":
            return dict(kind=kind, solver=solver, nx=rng.randint(11, 60), ny=rng.randint(17, 60), nz=1, surface=False)
        if solver == "3d2":
            return dict(kind=kind, solver=solver, nx=rng.randint(9, 38), ny=rng.randint(9, 19), nz=rng.randint(9, 19),
                        surface=rng.random() < 0.5)
        return dict(kind=kind, solver=solver, nx=rng.randint(20, 94), ny=rng.randint(7, 20), nz=rng.randint(20, 46),
                    surface=rng.random() < 0.5)
    if kind == "run":
        dim = rng.choice([2, 3, 3])
        n = _log_int(rng, 1500, 300000 if dim == 2 else 1000000)
        nx, ny, nz = _block(rng, n, dim)
        adaptive = rng.random() < 0.5
        mode = "launches" if adaptive else rng.choice(["launches", "graph", "persistent"])
        return dict(kind=kind, dim=dim, spacing=rng.choice([0.005, 0.01]), nx=nx, ny=ny, nz=nz,
                    ways=rng.choice([2, 4]) if dim == 3 else 2, adaptive=adaptive, steps=rng.randint(8, 20), mode=mode,
                    jitter=rng.choice([0.01, 0.05] if adaptive else [0.01, 0.05, 0.15]), surface=dim == 3 and rng.random() < 0.3)
    if kind == "batch":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, spacing=0.01, scenes=_log_int(rng, 5, 48), n_min=1024,
                    n_max=_log_int(rng, 2048, 16384), ways=rng.choice([2, 4]) if dim == 3 else 2,
                    steps=rng.randint(20, 60))
    dim = rng.choice([2, 3])
    nx, ny, nz = _block(rng, _log_int(rng, 800, 30000), dim)
    return dict(kind=kind, dim=dim, spacing=0.01, nx=nx, ny=ny, nz=nz, adaptive=rng.random() < 0.5,
                steps=rng.randint(10, 40), every=rng.choice([5, 10, 20]))


# ------------------------------------------------------------------ scenes
def _normal(seed, n, dim, sigma):
    r = np.random.default_rng(seed * 7919 + 13)
    return (sigma * r.standard_normal((n, dim))).astype(np.float32)


def _block_points(case, spacing, seed, jitter):
    dim = 2 if case.get("solver") == "2d" else case.get("dim", 3)
    counts = (case["nx"], case["ny"], case["nz"])[:dim]
    return scenes.lattice(counts, spacing, np.zeros(dim), seed, jitter=jitter)


def _grid_config(cfg, dim, cells):
    for a in range(dim):
        cfg.ncell[a] = int(cells[a])
        cfg.world[a] = float(np.float32(cells[a]) * np.float32(cfg.cell_size))
    if dim == 2:
        cfg.ncell[2], cfg.world[2] = 1, 0.0


def _si_config(case, cells):
    """Config of the SI workloads for the case's spacing, box and options."""
    dim, s = case["dim"], case["spacing"]
    if dim == 2:
        cfg = sph.preset(sph.PRESET_DAM_2D)
    elif s == 0.005:
        cfg = sph.preset(sph.PRESET_DAM_3D4)
    elif case["kind"] == "rollout":
        cfg = sph.preset(sph.PRESET_ROLLOUT_3D)
    else:
        cfg = sph.preset(sph.PRESET_DAM_3D2)
    for level, v in enumerate(_si_levels(dim, s, case.get("ways", 2))):
        for key, x in v.items():
            getattr(cfg, key)[level] = x
    cfg.split_ways = case.get("ways", 2)
    cfg.cell_size = cfg.kernel[0]
    cfg.close_r2 = float((np.float32(1e-3) * np.float32(cfg.kernel[0])) ** 2)
    cfg.time_step = _si_dt(case)
    cfg.compensated_positions = 1 if case["kind"] == "rollout" else 0
    _grid_config(cfg, dim, cells)
    cfg.use_split = cfg.use_merge = 1 if case.get("adaptive", True) else 0
    cfg.grid_every = 0
    for a in range(3):
        cfg.ndens[a] = 0
    if case.get("surface"):
        cfg.grid_every = 10
        cfg.dens_mul = 2
        cfg.den_size = float(np.float32(cfg.cell_size) / np.float32(2))
        for a in range(3):
            cfg.ndens[a] = 2 * cfg.ncell[a] + 1
    return cfg


def _si_dt(case):
    return (1e-4 if case["dim"] == 2 else 5e-5) * (case["spacing"] / 0.01)


def _si_levels(dim, s, ways):
    """Mass, lengths and kernel coefficients of the two levels, as the SI presets define them."""
    f = np.float32
    h0, m0 = f(2.0) * f(s), (f(1000.0) * f(s) * f(s) * f(s) if dim == 3 else f(1000.0) * f(s) * f(s))
    shrink = f(float(ways) ** (-1.0 / dim))
    out = []
    for m, h, r in ((m0, h0, f(0.5) * f(s)), (m0 / f(ways), h0 * shrink, f(0.5) * f(s) * shrink)):
        d, pi, rr = float(h), math.pi, float(r)
        k = (dict(poly6=315.0 / (64.0 * pi * d ** 9), spiky=-45.0 / (pi * d ** 6), visco=45.0 / (pi * d ** 6),
                  grad_poly6=-945.0 / (32.0 * pi * d ** 9), lapc_poly6=-945.0 / (8.0 * pi * d ** 9),
                  poly6_radius=315.0 / (64.0 * pi * rr ** 9)) if dim == 3 else
             dict(poly6=4.0 / (pi * d ** 8), spiky=-30.0 / (pi * d ** 5), visco=40.0 / (pi * d ** 5),
                  grad_poly6=-24.0 / (pi * d ** 8), lapc_poly6=-48.0 / (pi * d ** 8),
                  poly6_radius=4.0 / (pi * rr ** 8)))
        k.update(mass=m, kernel=h, kernel2=h * h, kernel6=d ** 6, radius=r)
        out.append({key: float(f(v)) for key, v in k.items()})
    return out


def _si_cells(case):
    """The box: twice the block along x, 1.5 times its height, one cell deeper."""
    n = (case["nx"], case["ny"], case["nz"])
    return [max(4, n[0]), max(4, -(-3 * n[1] // 4)), -(-n[2] // 2) + 1][:case["dim"]]


def _pinned(nbytes):
    return torch.zeros(nbytes, dtype=torch.uint8).pin_memory()


def _records(solver, pos, vel, level):
    """Page-locked reference-layout records of particles of one level."""
    rec = np.zeros(len(pos), sph.particle_dtype(solver.dim))
    rec["pos"], rec["vel"], rec["ev"], rec["level"] = pos, vel, vel, level
    up = _pinned(rec.nbytes)
    up.numpy()[:] = rec.view(np.uint8)
    return up


# ------------------------------------------------------------------ prepare
REF = {"2d": sph.PRESET_REF_2D, "3d2": sph.PRESET_REF_3D2, "3d4": sph.PRESET_REF_3D4}
REF_SPACING = {"2d": 0.5, "3d2": 0.8, "3d4": 0.5}   # the apps' own lattices, in their units (3d4 starts at level 2)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        cfg = sph.preset(REF[case["solver"]])
        cfg.use_split = cfg.use_merge = 1
        cfg.grid_every = 1 if case["surface"] else 0
        pos = _block_points(case, REF_SPACING[case["solver"]], seed, 0.05)
        vel = _normal(seed, len(pos), pos.shape[1], 0.2)
        cfg.max_particle = 4 * len(pos)
        st = dict(n=len(pos), steps=1)
    elif kind == "batch":
        cfg = _si_config(case, [4] * case["dim"])
        # layout, sizes and constants are the case's; jitter and velocities the seed's
        cfg, boxes, pos, vel, level, scene, _ = scenes.batch_scenes(cfg, case["scenes"], seed=4, n_min=case["n_min"],
                                                                    n_max=case["n_max"])
        pos = pos + _normal(seed + 1, len(pos), case["dim"], 0.01 * case["spacing"])
        vel = _normal(seed, len(pos), case["dim"], 0.1)
        s = sph.Solver(cfg)
        s.set_scenes(boxes)
        return dict(kind=kind, solver=s, steps=case["steps"], dim=case["dim"],
                    init=dict(pos=pos, vel=vel, ev=vel, level=level, scene=scene),
                    down=_pinned(case["ways"] * len(pos) * s.record_size))
    else:
        cfg = _si_config(case, _si_cells(case))
        pos, vel = _si_points(case, seed)
        cfg.max_particle = len(pos) * (4 if case["adaptive"] else 1)
        st = dict(n=len(pos), steps=case["steps"])
    s = sph.Solver(cfg)
    if kind == "rollout":
        origin, spacing, target = _loss_target(case, cfg, seed)
        return dict(kind=kind, solver=s, init=dict(pos=pos, vel=vel, ev=vel, level=np.ones(len(pos), np.uint32)),
                    n=len(pos), steps=case["steps"], every=case["every"], nodes=(GRID_LOSS,) * case["dim"],
                    origin=origin, spacing=spacing, target=target)
    mode = case.get("mode", "launches")
    s.set_graph(mode == "graph")
    s.set_persistent(mode == "persistent")
    st.update(kind=kind, solver=s, dim=s.dim, up=_records(s, pos, vel, 2 if case.get("solver") == "3d4" else 1), mesh=None,
              down=_pinned((cfg.split_ways if cfg.use_split else 1) * len(pos) * s.record_size))
    if case["surface"]:
        mv = sph.MeshView()
        mv.max_triangles = 500000
        tri = torch.zeros(6, mv.max_triangles, 3).pin_memory()
        for k, name in enumerate(("v0", "v1", "v2", "n0", "n1", "n2")):
            setattr(mv, name, ctypes.cast(tri[k].data_ptr(), ctypes.POINTER(ctypes.c_float)))
        st.update(mesh=mv, tri=tri)
    return st


def _si_points(case, seed):
    pos = _block_points(case, case["spacing"], seed, case.get("jitter", 0.01))
    return pos, _normal(seed, len(pos), case["dim"], 0.1)


def _loss_target(case, cfg, seed):
    """Loss grid over the box and a target density on it: the rest density
    with 20 % noise over the block, zero elsewhere."""
    dim = case["dim"]
    spacing = max(float(cfg.world[a]) for a in range(dim)) / GRID_LOSS
    origin = (0.5 * spacing,) * dim
    r = np.random.default_rng(seed * 104729 + 5)
    shape = (GRID_LOSS,) * dim                      # z, y, x: x fastest
    t = REST * (0.8 + 0.4 * r.random(shape))
    at = np.meshgrid(*[origin[a] + spacing * np.arange(GRID_LOSS) for a in range(dim)], indexing="ij")
    inside = np.ones(shape, bool)
    for a, count in enumerate((case["nx"], case["ny"], case["nz"])[:dim]):
        inside &= np.transpose(at[a]) < count * case["spacing"]
    return origin, spacing, np.where(inside, t, 0.0).astype(np.float32)


# ------------------------------------------------------------------ run
def _columns(records, dim):
    """The record fields as views of the download buffer (the whole of it:
    the records past the count stay zero)."""
    words = 18 if dim == 3 else 14
    f = records.view(torch.float32).view(-1, words)
    i = records.view(torch.int32).view(-1, words)
    out = {k: f[:, a * dim:(a + 1) * dim] for a, k in enumerate(("pos", "vel", "ev", "acc"))}
    b = 4 * dim
    out.update(dens=f[:, b], press=f[:, b + 1], energy=f[:, b + 2])
    out["surface"], out["level"] = (f[:, b + 3], i[:, b + 5]) if dim == 3 else (f[:, b + 4], i[:, b + 3])
    return out


def run(st):
    s = st["solver"]
    if st["kind"] == "rollout":
        s.set_state(st["init"])
        s.rollout_forward(st["steps"], st["every"])
        loss, grid = s.splat_loss(st["nodes"], st["origin"], st["spacing"], st["target"])
        g = s.rollout_backward(st["n"])
        # loss and parameter gradients are sums of 32-bit values: handed on in 32 bits, as to a torch optimiser
        return dict(loss=np.float32(loss), grid=grid, d_vel0=g["d_vel0"], d_pos0=g["d_pos0"],
                    d_params=g["d_params"].astype(np.float32))
    if st["kind"] == "batch":
        s.set_state(st["init"])
    else:
        s.write_particles_from(st["up"].data_ptr(), st["n"])
    s.step(st["steps"])
    n = s.read_particles_into(st["down"].data_ptr(), st["down"].numel())
    out = dict(count=n, **_columns(st["down"], st["dim"]))
    if st.get("mesh") is not None:
        mv = st["mesh"]
        rc = sph.lib().sph_extract_surface(s._h, ctypes.byref(mv))
        if rc:
            raise sph.SphError(rc, "sph_extract_surface")
        out.update(triangles=int(mv.num_triangles), vertices=st["tri"][:3], normals=st["tri"][3:])
    return out


# ------------------------------------------------------------------ work
def _batch_particles(case):
    """Particles of a batch (log-uniform sizes: their mean times the count)."""
    lo, hi = case["n_min"], case["n_max"]
    return int(case["scenes"] * (hi - lo) / math.log(hi / lo)) if hi > lo else case["scenes"] * lo


def work(case):
    """Per step and particle: position, velocity and half-step velocity read
    and written once, density, pressure, acceleration, energy and surface
    term written; records once up and once down; about 28 neighbours (2D 16)
    at 70 operations in the density, force and energy sums together.  A
    rollout's backward reads the step's state again and writes the adjoint."""
    dim = 2 if case.get("solver") == "2d" else case.get("dim", 3)
    n = _batch_particles(case) if case["kind"] == "batch" else case["nx"] * case["ny"] * case["nz"]
    steps = case.get("steps", 1)
    state, record = 4 * 3 * dim, 72 if dim == 3 else 56
    pairs = 28 if dim == 3 else 16
    nbytes = n * (steps * 2 * state + 2 * record)
    flops = n * steps * pairs * 70.0
    if case["kind"] == "rollout":
        nbytes, flops = 2 * nbytes, 3 * flops
    return {"bytes": float(nbytes), "flops": float(flops)}


# ------------------------------------------------------------------ 64-bit values
class _Exact:
    """The SI step without adaptivity in 64 bits (one level, plain torch)."""

    def __init__(self, case):
        self.dim = case["dim"]
        self.k = _si_levels(self.dim, case["spacing"], case.get("ways", 2))[0]
        self.dt = float(np.float32(_si_dt(case)))
        self.close = float((np.float32(1e-3) * np.float32(self.k["kernel"])) ** 2)
        self.cells = _si_cells(case)
        self.h = self.k["kernel"]
        self.world = [float(np.float32(c) * np.float32(self.h)) for c in self.cells]
        self.mu, self.gas = 0.1, 3.0

    def cell_of(self, x):
        # the cell of a position is decided on its 32-bit value, as the library decides it
        top = torch.tensor([c - 1 for c in self.cells], device=x.device)
        q = torch.floor(x.float() / torch.tensor(self.h, dtype=torch.float32, device=x.device)).long()
        return torch.minimum(torch.clamp(q, min=0), top)

    def pairs(self, x, reach):
        """Directed pairs (i, j), j != i, closer than reach (<= the cell edge times 1.02)."""
        with torch.no_grad():
            edge = 1.05 * self.h
            top = [int(w / edge) + 2 for w in self.world]
            q = torch.clamp(torch.floor(x / edge).long() + 1, min=0)
            q = torch.minimum(q, torch.tensor([t + 1 for t in top], device=x.device))
            size = [t + 3 for t in top]
            key = q[:, 0]
            for a in range(1, self.dim):
                key = key + q[:, a] * math.prod(size[:a])
            order = torch.argsort(key, stable=True)
            total = math.prod(size)
            counts = torch.bincount(key, minlength=total)
            first = torch.cumsum(counts, 0) - counts
            most = int(counts.max())
            got = []
            for off in np.ndindex(*(3,) * self.dim):
                d = sum((o - 1) * math.prod(size[:a]) for a, o in enumerate(off))
                near = torch.clamp(key + d, 0, total - 1)
                b, c = first[near], counts[near]
                for u in range(most):
                    i = torch.nonzero(c > u).squeeze(1)
                    j = order[b[i] + u]
                    keep = ((x[i] - x[j]) ** 2).sum(1) < reach * reach
                    keep &= i != j
                    got.append(torch.stack([i[keep], j[keep]]))
            return torch.cat(got, 1)

    def density(self, x, pr):
        k, h2 = self.k, self.k["kernel2"]
        i, j = pr
        r2 = ((x[i] - x[j]) ** 2).sum(1)
        w = torch.clamp(h2 - r2, min=0.0) ** 3
        rho = torch.zeros(len(x), dtype=x.dtype, device=x.device).index_add(0, i, w)
        rho = k["mass"] * k["poly6"] * (rho + k["kernel6"])
        return rho, self.gas * ((rho / REST) ** 3 - 1.0)

    def step(self, x, v, ev, outputs=False):
        k, h, m = self.k, self.h, self.k["mass"]
        i, j = pr = self.pairs(x, (1.02 if outputs else 1.0) * h)
        rho, p = self.density(x, pr)
        d = x[i] - x[j]
        r2 = (d * d).sum(1)
        inside = (r2 < k["kernel2"]) & (r2 >= self.close)
        r = torch.sqrt(torch.where(inside, r2, torch.ones_like(r2)))
        q = torch.where(inside, h - r, torch.zeros_like(r))
        a, vol = p / (rho * rho), m / rho
        # both kernels of a pair are the same: 0.5 * (term + term)
        tp = m * m * (a[i] + a[j]) * k["spiky"] * q * q / r
        tv = vol[i] * vol[j] * self.mu * k["visco"] * q
        f = torch.zeros_like(x).index_add(0, i, (ev[j] - ev[i]) * tv[:, None] - d * tp[:, None])
        out = None
        if outputs:
            u = torch.where(inside, k["kernel2"] - r2, torch.zeros_like(r2))
            grad = torch.zeros_like(x).index_add(0, i, d * (-k["grad_poly6"] * vol[j] * u * u)[:, None])
            out = dict(dens=rho, press=p, acc=f, surface=torch.sqrt((grad * grad).sum(1)))
        g = torch.zeros(self.dim, dtype=x.dtype, device=x.device)
        g[1] = float(np.float32(GRAVITY))
        v = v + (f / m + g) * self.dt
        x0, x = x, x + v * self.dt
        xs, vs = [], []
        for c in range(self.dim):
            hi, lo = self.world[c] - k["radius"], k["radius"]
            over, under = x[:, c] >= hi, x[:, c] < lo
            xs.append(torch.where(over, torch.full_like(x[:, c], hi), torch.where(under, torch.full_like(x[:, c], lo), x[:, c])))
            vs.append(torch.where(over | under, -0.5 * v[:, c], v[:, c]))
        x, v = torch.stack(xs, 1), torch.stack(vs, 1)
        ev = (ev + v) / 2.0
        if outputs:
            out.update(energy=self.energy(x0, x, v, pr))
        return x, v, ev, out

    def energy(self, x0, x, v, pr):
        """Wavelet energy of the moved particles over the cells of the step's start."""
        i, j = pr
        near = ((self.cell_of(x[i]) - self.cell_of(x0[j])).abs() <= 1).all(1)
        d = x[i] - x[j]
        r2 = (d * d).sum(1)
        ok = near & (r2 < self.k["kernel2"]) & (r2 >= self.close)
        i, j, d = i[ok], j[ok], d[ok] / self.h
        amp = 2.0 / (3.141592 ** 0.25 * math.sqrt(6.0))
        w = amp * (d * d / 4.0 - 1.0) * torch.exp(-d * d / 8.0 * math.log(2.718281))
        ts = torch.zeros_like(x).index_add(0, i, w)
        tv = torch.zeros_like(x).index_add(0, i, v[j] * w) / math.sqrt(self.h)
        t = tv / ts
        return 0.5 * (t[:, :2] ** 2).sum(1)      # the x and y components, as the reference sums them


def exact(case, seed):
    """64-bit values of the cases without splits.  Where particles split or
    merge, the layout follows yes/no decisions on 32-bit sums, which a 64-bit
    trajectory takes differently for some particles: no value."""
    if case["kind"] not in ("run", "rollout") or case["adaptive"]:
        return None
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > (12 << 20):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pos, vel = _si_points(case, seed)
    x, v = (torch.from_numpy(a).to(dev, torch.float64) for a in (pos, vel))
    e = _Exact(case)
    if case["kind"] == "run":
        ev = v
        for q in range(case["steps"]):
            x, v, ev, out = e.step(x, v, ev, outputs=q == case["steps"] - 1)
        mesh = dict(triangles=None, vertices=None, normals=None) if case["surface"] else {}
        return dict(count=None, pos=x, vel=v, ev=ev, level=None, **out, **mesh)
    x0, v0 = x.requires_grad_(True), v.requires_grad_(True)
    ev = v0.detach()            # the state's ev field is not the velocity variable
    e.mu = torch.tensor(float(np.float32(0.1)), dtype=torch.float64, device=dev, requires_grad=True)
    e.gas = torch.tensor(3.0, dtype=torch.float64, device=dev, requires_grad=True)
    x, v = x0, v0
    for q in range(case["steps"]):
        x, v, ev, _ = e.step(x, v, ev)
    cfg = sph.Config()          # only the box of the loss grid
    for a in range(e.dim):
        cfg.world[a] = e.world[a]
    origin, spacing, target = _loss_target(case, cfg, seed)
    grid = _splat(e, x, origin, spacing)
    loss = ((grid - torch.from_numpy(target).to(dev, torch.float64).reshape(-1)) ** 2).mean()
    gx, gv, gm, gk = torch.autograd.grad(loss, (x0, v0, e.mu, e.gas))
    return dict(loss=loss.detach(), grid=grid.detach(), d_vel0=gv, d_pos0=gx,
                d_params=torch.stack([gm, gk]).reshape(1, 2))


def _splat(e, x, origin, spacing):
    """Density on the loss grid's nodes, x fastest."""
    f = np.float32
    axes = [torch.tensor([float(f(float(f(origin[a])) + u * float(f(spacing)))) for u in range(GRID_LOSS)],
                         dtype=torch.float64, device=x.device) for a in range(e.dim)]
    reach = int(e.h / spacing) + 2
    base = torch.floor((x.detach() - origin[0]) / spacing).long()
    grid = torch.zeros(GRID_LOSS ** e.dim, dtype=torch.float64, device=x.device)
    for off in np.ndindex(*(2 * reach + 1,) * e.dim):
        q = base + torch.tensor([o - reach for o in off], device=x.device)
        ok = ((q >= 0) & (q < GRID_LOSS)).all(1)
        q, y = q[ok], x[ok]
        r2 = sum((y[:, a] - axes[a][q[:, a]]) ** 2 for a in range(e.dim))
        w = e.k["mass"] * e.k["poly6"] * torch.clamp(e.k["kernel2"] - r2, min=0.0) ** 3
        at = sum(q[:, a] * GRID_LOSS ** a for a in range(e.dim))
        grid = grid.index_add(0, at, w)
    return grid
