"""Performance cases of the framework: what its users call, over the range of sizes they call it with.

Every case goes through a public entry point: ``SolverPBF/SolverDFSPH/SolverWCSPH.step``, a ``FrameGraph``, a batched
model on a ``WorldGrid``, ``DiffWCSPH.rollout`` with its backward pass, ``ParticleSeparation.apply`` and
``HashGrid.build`` / ``tables``.  Inputs are made on the GPU from a seed: a disordered water column in the reference
dam-break tank (jittered lattice at rest spacing, a collapsing shear flow plus noise), or a box filled by a jittered
body-centred lattice.  ``exact`` evaluates the same step in float64 with plain torch.
"""

import math
import random
from types import SimpleNamespace

import numpy as np
import torch

from fluid_simulation_b200.apic import ParticleSeparation
from fluid_simulation_b200.batch import Batch, batched_model, make_batch
from fluid_simulation_b200.dam_break import material, solver_config
from fluid_simulation_b200.diff import DiffWCSPH
from fluid_simulation_b200.graph import FrameGraph
from fluid_simulation_b200.newton_shim import HashGrid, model_from_arrays
from fluid_simulation_b200.scene import DEFAULT_SPEC, ParticleScene
from fluid_simulation_b200.solver import SolverDFSPH, SolverPBF, SolverWCSPH

DEV = "cuda:0"
SOLVERS = {"pbf": SolverPBF, "dfsph": SolverDFSPH, "wcsph": SolverWCSPH}
WALLS = (1.2, 0.28, 0.6)  # bound_width, bound_height, bound_length of the dam-break tank


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # one substep of a tiny interactive scene: launches and latency are everything
        dict(name="pbf_4k", kind="step", method="pbf", n=4079),
        # the reference's CPU-sized dam break, one WCSPH substep
        dict(name="wcsph_10k", kind="step", method="wcsph", n=9936),
        # a display frame (four PBF substeps) replayed as one CUDA graph from a given start
        dict(name="pbf_frame_20k", kind="frame", method="pbf", n=19997, substeps=4),
        # a preview-sized DFSPH substep, warm-started from the previous step's kappas
        dict(name="dfsph_30k", kind="step", method="dfsph", n=30011, warm=True),
        # PBF with everything on: artificial pressure, cohesion, viscosity, the class's ten iterations
        dict(name="pbf_scorr_100k", kind="step", method="pbf", n=100003, scorr=True, iterations=10),
        # the reference's own dam-break size, PBF and DFSPH with the harness's settings
        dict(name="pbf_400k", kind="step", method="pbf", n=401856),
        dict(name="dfsph_400k", kind="step", method="dfsph", n=401856),
        # the neighbour-search stress: a 1.6 m box full of fluid
        dict(name="wcsph_4m", kind="lattice", method="wcsph", cells=128),
        # many independent scenes of uneven size in one model (training data, parameter sweeps)
        dict(name="pbf_batch_64", kind="batch", method="pbf", scenes=64, n_lo=2000, n_hi=100000, draw=3),
        # a differentiable rollout: forward and backward, gradients of every input
        dict(name="wcsph_grad_50k", kind="grad", n=50232, steps=20, every=10),
        # the APIC solver's particle separation, two iterations
        dict(name="separation_400k", kind="separation", n=401856),
        # the neighbour grid alone, with its tables read back on the device
        dict(name="grid_1m", kind="grid", n=1000003),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["step"] * 7 + ["frame", "lattice", "batch", "grad", "separation", "grid"])
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if kind == "step":
        method = rng.choice(["pbf", "dfsph", "wcsph"])
        c = dict(kind=kind, method=method, n=size(4000, 600000 if method == "dfsph" else 1000000))
        if method == "pbf" and rng.random() < 0.3:
            c.update(n=size(4000, 400000), scorr=True, iterations=rng.randint(2, 10))
        if method == "dfsph" and rng.random() < 0.3:
            c.update(warm=True)
        return c
    if kind == "frame":
        return dict(kind=kind, method="pbf", n=size(4000, 200000), substeps=2 * rng.randint(1, 3))
    if kind == "lattice":
        return dict(kind=kind, method="wcsph", cells=size(24, 120))
    if kind == "batch":
        return dict(kind=kind, method=rng.choice(["pbf", "wcsph", "dfsph"]), scenes=rng.randint(4, 48), n_lo=2000,
                    n_hi=size(4000, 60000), draw=rng.randint(4, 1 << 20))
    if kind == "grad":
        return dict(kind=kind, n=size(4000, 50000), steps=rng.randint(3, 20), every=rng.randint(2, 10))
    if kind == "separation":
        return dict(kind=kind, n=size(10000, 1000000))
    return dict(kind=kind, n=size(4000, 4000000))


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _column(n, seed):
    """(x, v, spacing): n particles of a water column in the tank's low-x corner."""
    lo = (-1.17, -0.25, 0.03)
    ext = (0.702, 0.5, 0.8208)
    spacing = (ext[0] * ext[1] * ext[2] / n) ** (1.0 / 3.0)
    ry, rz = max(2, int(ext[1] / spacing)), max(2, int(ext[2] / spacing))
    k = torch.arange(n, device=DEV, dtype=torch.int64)
    ijk = torch.stack([k // (ry * rz), k // rz % ry, k % rz], 1)  # the last layer may be ragged
    g = _gen(seed)
    jitter = 0.2 * (2.0 * torch.rand(n, 3, device=DEV, generator=g, dtype=torch.float64) - 1.0)
    x = torch.tensor(lo, device=DEV, dtype=torch.float64) + (ijk + 0.5 + jitter) * spacing
    v = 0.1 * torch.randn(n, 3, device=DEV, generator=g, dtype=torch.float64)
    v[:, 0] += 0.8 * (x[:, 0] + 1.2) / 0.7
    v[:, 2] -= 0.5 * x[:, 2]
    return x.float().contiguous(), v.float().contiguous(), float(spacing)


def _lattice(cells, seed):
    """(x, v, spacing): 2 cells^3 particles of a body-centred lattice filling a box at 9.9 mm rest spacing."""
    a = 0.0125
    box = cells * a
    c = (torch.arange(cells, device=DEV, dtype=torch.float64) + 0.25) * a
    z, y, x = torch.meshgrid(c, c - 0.5 * box, c - 0.5 * box, indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    p = torch.cat([p, p + 0.5 * a])
    d = a / 2.0 ** (1.0 / 3.0)
    g = _gen(seed)
    p += 0.1 * d * (2.0 * torch.rand(p.shape, device=DEV, generator=g, dtype=torch.float64) - 1.0)
    v = 0.2 * torch.randn(p.shape, device=DEV, generator=g, dtype=torch.float64)
    return p.float().contiguous(), v.float().contiguous(), d


def _scene(spacing):
    return ParticleScene(DEFAULT_SPEC, None, 1000.0 * spacing ** 3, 0.5 * spacing, spacing ** 3, spacing)


def _batch(case) -> Batch:
    return make_batch(case["scenes"], seed=case["draw"], n_lo=case["n_lo"], n_hi=case["n_hi"])


def _batch_inputs(case, seed):
    b = _batch(case)
    rng = np.random.default_rng(seed)
    for s in b.scenes:
        w = np.array([s.walls[0], s.walls[1], 2.0 * s.walls[2]])
        x = s.x + 0.2 * b.spacing * rng.uniform(-1.0, 1.0, s.x.shape)
        s.x = np.clip(x, [-w[0], -w[1], 0.0], w).astype(np.float32)
    v = (0.1 * rng.standard_normal((b.total, 3))).astype(np.float32)
    return b, v


def _problem(case, seed):
    """The step's inputs and settings, from the case and the seed alone."""
    p = SimpleNamespace(kind=case["kind"], method=case.get("method", "wcsph"), world=None, stiffness=None, batch=None)
    if case["kind"] == "batch":
        p.batch, v = _batch_inputs(case, seed)
        p.x = torch.as_tensor(p.batch.positions(), device=DEV)
        p.v = torch.as_tensor(v, device=DEV)
        p.spacing = p.batch.spacing
        p.world = torch.as_tensor(p.batch.world(), device=DEV)
        walls = torch.tensor([s.walls for s in p.batch.scenes], dtype=torch.float64, device=DEV)
        p.walls = walls.float().double()[p.world.long()]
        p.viscosity = torch.as_tensor(p.batch.per_particle("viscosity"), device=DEV).double()
        p.stiffness = torch.as_tensor(p.batch.per_particle("stiffness"), device=DEV).double()
    else:
        p.x, p.v, p.spacing = (_lattice(case["cells"], seed) if case["kind"] == "lattice"
                               else _column(case["n"], seed))
        walls = (0.5 * case["cells"] * 0.0125,) * 3 if case["kind"] == "lattice" else WALLS
        p.walls = torch.tensor(walls, dtype=torch.float64, device=DEV).float().double()
    p.n = p.x.shape[0]
    scene = _scene(p.spacing)
    p.config = solver_config(p.method, scene)
    p.attributes = dict(material(p.method, scene), particle_mask=0)
    if case["kind"] == "lattice":
        p.config.bound_width, p.config.bound_height, p.config.bound_length = walls
    if case.get("scorr"):
        p.config.scorr_k, p.config.scorr_n, p.config.scorr_q = 1.0e-4, 4.0, 0.3
        p.config.max_iterations = int(case["iterations"])
        p.attributes.update(surface_tension=0.01, viscosity=0.005)
    if case.get("warm"):
        p.config.warm_start = True
    p.mass, p.radius = scene.mass, scene.radius
    h = 2.0 * p.spacing
    sound = math.sqrt(250000.0 * 7.0 / 1000.0)
    speed = 2.0  # above the inputs' largest velocity component: the time step is known before the call
    p.dt = {"pbf": 1.0 / 240.0, "dfsph": min(1.0 / 240.0, 0.4 * p.spacing / speed),
            "wcsph": 0.25 * h / (sound * 1.1 + speed)}[p.method]
    return p


def _solver(p):
    cls = SOLVERS[p.method]
    if p.batch is not None:
        model = batched_model(p.batch, cls, device=DEV, v=p.v)
        p.config.particle_radius = p.batch.radius
    else:
        model = model_from_arrays(p.x, p.v, p.mass, device=DEV, radius=p.radius, gravity=((0.0, 0.0, -10.0),),
                                  attributes=p.attributes, solver_cls=cls)
    return model, cls(model, p.config)


def prepare(case, seed):
    if case["kind"] == "grid":
        x, _, spacing = _column(case["n"], seed)
        grid = HashGrid(128, 128, 128, device=DEV)
        grid.reserve(case["n"])
        return SimpleNamespace(kind="grid", x=x, grid=grid, radius=2.0 * spacing)
    if case["kind"] == "separation":
        x, _, spacing = _column(case["n"], seed)
        model = model_from_arrays(x, torch.zeros_like(x), 1000.0 * spacing ** 3, device=DEV, radius=0.5 * spacing)
        sep = ParticleSeparation(model, ParticleSeparation.Config(bound_lo=DEFAULT_SPEC.bound_lo,
                                                                  bound_hi=DEFAULT_SPEC.bound_hi))
        return SimpleNamespace(kind="separation", sep=sep, x=x, state=model.state())
    p = _problem(case, seed)
    model, solver = _solver(p)
    s = SimpleNamespace(kind=case["kind"], method=p.method, model=model, solver=solver, dt=p.dt)
    if case["kind"] == "grad":
        s.sim = DiffWCSPH(model, p.config, p.dt, checkpoint_every=case["every"])
        full = lambda v: torch.full((p.n,), float(v), device=DEV, requires_grad=True)  # noqa: E731
        s.inputs = [p.x.clone().requires_grad_(), p.v.clone().requires_grad_(), full(p.attributes["stiffness"]),
                    full(p.attributes["viscosity"]), full(1000.0)]
        s.target = p.x + torch.tensor([0.3, 0.0, 0.0], device=DEV)
        s.steps = case["steps"]
        return s
    s.a, s.b = model.state(), model.state()
    if case["kind"] == "frame":
        s.x, s.v = p.x, p.v
        s.graph = FrameGraph(solver, s.a, s.b, p.dt, substeps=case["substeps"])
    return s


# -------------------------------------------------------------------- runs --
def _outputs(s, state):
    out = dict(vars(state.sph), x=state.particle_q, v=state.particle_qd, accel=s.solver._particle_accel)
    out.pop("step_displacement", None)  # registered for the user, written by no step
    if s.method == "pbf":
        out["x_pred"] = s.solver._x_pred
    return out


def run(s):
    if s.kind == "grid":
        s.grid.build(s.x, s.radius)
        return s.grid.tables()
    if s.kind == "separation":
        s.state.particle_q.copy_(s.x)
        s.sep.apply(s.state)
        return s.state.particle_q
    if s.kind == "grad":
        x, v = s.sim.rollout(*s.inputs, s.steps)
        loss = ((x - s.target) ** 2).sum(1).mean()
        return dict(x=x, v=v, loss=loss, grads=torch.autograd.grad(loss, s.inputs))
    if s.kind == "frame":  # from a given start, as a user who resets a scene and plays it
        s.a.particle_q.copy_(s.x)
        s.a.particle_qd.copy_(s.v)
        return _outputs(s, s.graph.replay())
    s.solver.step(s.a, s.b, None, None, s.dt)
    return _outputs(s, s.b)


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes: the step's inputs read once and its outputs written once.  Flops: the pair terms of the passes that the
    method prescribes, at about 34 neighbours within the support."""
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["draw"])
        n = float(np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), case["scenes"])).sum())
    else:
        n = float(2 * case["cells"] ** 3 if case["kind"] == "lattice" else case["n"])
    pairs = 34.0 * n
    if case["kind"] == "grid":
        return dict(bytes=n * (12 + 8) + 2.0 * 4 * 128 ** 3, flops=6.0 * n)
    if case["kind"] == "separation":  # x in and out, flags; about 6 neighbours closer than the rest distance
        return dict(bytes=28.0 * n, flops=2 * 6.0 * n * 20)
    method = case.get("method", "wcsph")
    attributes = 4.0 * (4 + 3)  # mass, flags, mask, world; rest density, surface tension, viscosity
    if method == "pbf":  # x, v in; x, v, rho, lambda, count, delta, accel, x_pred out
        it = case.get("iterations", 4)
        per = 24 + attributes + 24 + 12 + 36
        flops = pairs * (2 * 14 + 30 + it * (30 + 25) + 18)
    elif method == "dfsph":  # x, v in; x, v, rho, factor, rho*, rate, kappas, count, v*, accel out
        per = 24 + attributes + 24 + 28 + 24
        flops = pairs * (2 * 30 + 30 + 17 * (25 + 22))
    else:  # x, v, stiffness, exponent in; x, v, rho, p, accel out
        per = 24 + attributes + 8 + 24 + 8 + 12
        flops = pairs * (16 + 40)
    if case["kind"] == "frame":
        return dict(bytes=n * per, flops=flops * case["substeps"])
    if case["kind"] == "grad":  # three parameter fields in, x, v and five gradients out
        return dict(bytes=n * (24 + attributes + 8 + 24 + 24 + 12 + 12), flops=case["steps"] * (flops + pairs * 150))
    return dict(bytes=n * per, flops=flops)


# ------------------------------------------------------------------- exact --
def _pairs(q, b, h, world=None):
    """Chunks (i, j, r^2) of the pairs with |q_i - q_j| <= h among the candidates of a grid of cells trunc(x / h) that
    binned the particles at b and is queried at q; also the number of candidates of each particle."""
    n = q.shape[0]
    cb = torch.trunc(b / h).long()
    lo, hi = torch.trunc((q - h) / h).long(), torch.trunc((q + h) / h).long()
    c0, c1 = cb.amin(0), cb.amax(0)
    dim = c1 - c0 + 1
    w = torch.zeros(n, dtype=torch.long, device=q.device) if world is None else world.long()
    key = lambda c: ((w * dim[2] + c[:, 2] - c0[2]) * dim[1] + c[:, 1] - c0[1]) * dim[0] + c[:, 0] - c0[0]  # noqa: E731
    skey, order = torch.sort(key(cb), stable=True)
    chunks, count = [], torch.zeros(n, dtype=torch.long, device=q.device)
    for k in range(27):
        c = lo + torch.tensor([k % 3, k // 3 % 3, k // 9], device=q.device)
        ok = ((c <= hi) & (c >= c0) & (c <= c1)).all(1)
        kk = torch.where(ok, key(c), -1)
        s, e = torch.searchsorted(skey, kk), torch.searchsorted(skey, kk, right=True)
        m = torch.where(ok, e - s, 0)
        count += m
        i = torch.repeat_interleave(torch.arange(n, device=q.device), m)
        first = torch.cumsum(m, 0) - m
        j = order[(s - first)[i] + torch.arange(i.shape[0], device=q.device)]
        r2 = ((q[i] - q[j]) ** 2).sum(1)
        near = r2 <= h * h
        chunks.append((i[near], j[near], r2[near]))
    return chunks, count


def _sum(n, chunks, term, width=None):
    out = torch.zeros((n,) if width is None else (n, width), dtype=torch.float64, device=DEV)
    for i, j, r2 in chunks:
        out.index_add_(0, i, term(i, j, r2))
    return out


def _cubic(h):
    k = 8.0 / (math.pi * h ** 3)

    def w(r):
        q = r / h
        near, far = k * (6.0 * q ** 3 - 6.0 * q * q + 1.0), 2.0 * k * (1.0 - q).clamp(min=0.0) ** 3
        return torch.where(q <= 0.5, near, far)

    def gs(r):  # grad W = gs(r) d
        q = r / h
        inv = 1.0 / (r.clamp(min=1.0e-30) * h)
        near, far = 6.0 * k * q * (3.0 * q - 2.0) * inv, -6.0 * k * (1.0 - q) ** 2 * inv
        return torch.where((r > 1.0e-5) & (q <= 1.0), torch.where(q <= 0.5, near, far), torch.zeros_like(r))
    return w, gs


def _box(p, inset=0.0):
    """(lo, hi) of the tank, per particle where the scenes have tanks of their own."""
    w = p.walls
    lo = torch.stack([-w[..., 0] + inset, -w[..., 1] + inset, torch.zeros_like(w[..., 2]) + inset], -1)
    hi = torch.stack([w[..., 0] - inset, w[..., 1] - inset, 2.0 * w[..., 2] - inset], -1)
    return lo, hi


def _f32(v):
    return float(np.float32(v))


def _material(p, name):
    v = getattr(p, name, None)
    return v if v is not None else torch.full((p.n,), _f32(p.attributes[name]), dtype=torch.float64, device=DEV)


def _exact_pbf(p, x, v):
    c, n, h, dt, m = p.config, p.n, _f32(2.0 * p.spacing), _f32(p.dt), _f32(p.mass)
    rho0, mu, gamma = 1000.0, _material(p, "viscosity"), _f32(p.attributes["surface_tension"])
    kw, kg, rp = 315.0 / (64.0 * math.pi * h ** 9), -45.0 / (math.pi * h ** 6), _f32(p.radius)
    lo, hi = _box(p, rp)
    w = lambda r2: torch.where(r2 < h * h, kw * (h * h - r2) ** 3, torch.zeros_like(r2))  # noqa: E731

    def gs(r2):
        r = r2.sqrt()
        return torch.where((r > 1.0e-6) & (r < h), kg * (h - r) ** 2 / r.clamp(min=1.0e-30), torch.zeros_like(r))
    x_in = x
    vp = v + dt * torch.tensor([0.0, 0.0, -10.0], dtype=torch.float64, device=DEV)
    x = torch.minimum(torch.maximum(x + dt * vp, lo), hi)
    bins = x
    near, _ = _pairs(x, bins, h, p.world)
    rho = _sum(n, near, lambda i, j, r2: m * w(r2))

    def force(i, j, r2):
        d = x[i] - x[j]
        a = -(gamma / m) * m * w(r2.clamp(min=rp * rp)) * (i != j)
        vd = ((vp[i] - vp[j]) * d).sum(1)
        a = a + 10.0 * mu[i] * m / rho[j].clamp(min=1.0e-6) * vd / (r2 + 0.01 * h * h) * gs(r2)
        return a[:, None] * d
    accel = _sum(n, near, force, 3)
    x = torch.minimum(torch.maximum(x + dt * dt * accel, lo), hi)
    wdq = 315.0 / (64.0 * math.pi * h ** 9) * (h * h * (1.0 - c.scorr_q ** 2)) ** 3
    for it in range(c.max_iterations):
        near, _ = _pairs(x, bins, h, p.world)
        g = lambda i, j, r2: (-(m / rho0) * gs(r2))[:, None] * (x[i] - x[j])  # noqa: E731,B023
        rho = _sum(n, near, lambda i, j, r2: m * w(r2))
        grad = _sum(n, near, g, 3)
        sq = _sum(n, near, lambda i, j, r2: (g(i, j, r2) ** 2).sum(1)) + (grad ** 2).sum(1)
        cnt = _sum(n, near, lambda i, j, r2: ((i != j) & (r2 < h * h)).double())
        lam = -(rho / rho0 - 1.0).clamp(min=0.0) / (sq + c.lambda_epsilon)
        lam = torch.where(cnt < c.min_neighbors_for_lambda, torch.zeros_like(lam), lam)

        def push(i, j, r2):
            s = -c.scorr_k * (w(r2) / wdq) ** c.scorr_n if c.scorr_k else 0.0
            return ((lam[i] + lam[j] + s) * m * gs(r2))[:, None] * (x[i] - x[j])  # noqa: B023
        dp = _sum(n, near, push, 3) / rho0
        if c.max_delta_position > 0.0:
            big = dp.norm(dim=1, keepdim=True)
            dp = torch.where(big > c.max_delta_position, dp * (c.max_delta_position / big.clamp(min=1.0e-12)), dp)
        x = x + dp
        if it == c.max_iterations - 1:
            x = torch.minimum(torch.maximum(x, lo), hi)
    near, _ = _pairs(x, bins, h, p.world)
    rho = _sum(n, near, lambda i, j, r2: m * w(r2))
    u = (x - x_in) / dt
    u = u + c.xsph_c * _sum(n, near, lambda i, j, r2: (m / rho[j].clamp(min=1.0e-6) * w(r2))[:, None] * (u[j] - u[i]), 3)
    out = torch.where((x < lo) & (u < 0) | (x > hi) & (u > 0), u * c.boundary_damping, u)
    return dict(rho=rho, pbf_lambda=lam, neighbor_count=None, delta_p=dp, x=torch.minimum(torch.maximum(x, lo), hi),
                v=out, accel=accel, x_pred=x)


def _non_pressure(p, near, x, v, rho, m, h):
    """Viscosity, cohesion and gravity (WCSPH and DFSPH)."""
    w, gs = _cubic(h)
    mu, gamma, rp = _material(p, "viscosity"), _f32(p.attributes["surface_tension"]), _f32(p.radius)

    def term(i, j, r2):
        d = x[i] - x[j]
        r = r2.sqrt()
        vd = ((v[i] - v[j]) * d).sum(1)
        a = 10.0 * mu[i] * m / rho[j].clamp(min=1.0e-6) * vd / (r2 + 0.01 * h * h) * gs(r)
        return (a - (gamma / m) * m * w(r.clamp(min=rp)))[:, None] * d
    return _sum(p.n, near, term, 3) + torch.tensor([0.0, 0.0, -10.0], dtype=torch.float64, device=DEV)


def _exact_dfsph(p, x, v):
    c, n, h, dt, m = p.config, p.n, _f32(2.0 * p.spacing), _f32(p.dt), _f32(p.mass)
    w, gs = _cubic(h)
    lo, hi = _box(p)
    nw = 1 if p.world is None else int(p.world.max()) + 1
    wid = torch.zeros(n, dtype=torch.long, device=DEV) if p.world is None else p.world.long()
    per = torch.bincount(wid, minlength=nw).double()

    def density_factor(x):
        near, cand = _pairs(x, x, h, p.world)
        near = [(i, j, r2, r2.sqrt(), gs(r2.sqrt())) for i, j, r2 in near]
        rho, grad, sq = (torch.zeros(s, dtype=torch.float64, device=DEV) for s in ((n,), (n, 3), (n,)))
        for i, j, r2, r, s in near:
            rho.index_add_(0, i, m * w(r))
            g = (m * s)[:, None] * (x[i] - x[j])
            grad.index_add_(0, i, g)
            sq.index_add_(0, i, (g ** 2).sum(1))
        den = (grad ** 2).sum(1) + sq
        f = torch.where((cand - 1 < c.min_neighbors_for_factor) | (den < 1.0e-6), torch.zeros_like(den), 1.0 / den)
        return near, rho, f

    def rate(near, x, u):
        d = torch.zeros(n, dtype=torch.float64, device=DEV)
        for i, j, r2, r, s in near:
            d.index_add_(0, i, m * s * ((u[i] - u[j]) * (x[i] - x[j])).sum(1))
        return d

    def correct(near, x, u, kappa, rho):
        k = kappa / rho.clamp(min=1.0e-6)
        dv = torch.zeros(n, 3, dtype=torch.float64, device=DEV)
        for i, j, r2, r, s in near:
            dv.index_add_(0, i, (m * (k[i] + k[j]) * s)[:, None] * (x[i] - x[j]))
        return u - dt * dv
    out = {}
    near, rho, f = density_factor(x)
    accel = _non_pressure(p, [t[:3] for t in near], x, v, rho, m, h)
    u = v + dt * accel

    def solve(near, x, u, rho, f, iterations, eta, divergence):
        kappa = torch.zeros(n, dtype=torch.float64, device=DEV)
        live = torch.ones(nw, dtype=torch.bool, device=DEV)
        d = rs = None
        for it in range(iterations):
            nd = rate(near, x, u)
            on = live[wid]
            d = nd if d is None else torch.where(on, nd, d)
            if divergence:
                err = d.clamp(min=0.0)
                new = (err * rho * f / dt).clamp(max=c.max_kappa_v)
            else:
                nrs = rho + dt * nd
                rs = nrs if rs is None else torch.where(on, nrs, rs)
                err = (rs - 1000.0).clamp(min=0.0)
                new = (err / (dt * dt) * f).clamp(max=c.max_kappa)
            res = torch.zeros(nw, dtype=torch.float64, device=DEV).index_add_(0, wid, err) / per
            if it > 0:
                live = live & (res > eta)
            on = live[wid]
            kappa = torch.where(on, new, kappa)
            u = torch.where(on[:, None], correct(near, x, u, new, rho), u)
        return u, kappa, d, rs
    u, out["kappa"], _, out["rho_star"] = solve(near, x, u, rho, f, c.max_rho_iterations, c.eta_density, False)
    x = x + dt * u
    near, rho, f = density_factor(x)
    u, out["kappa_v"], out["d_rho_dt"], _ = solve(near, x, u, rho, f, c.max_vel_iterations, c.eta_divergence, True)
    hit = (x < lo) | (x > hi)
    return dict(out, rho=rho, factor=f, neighbor_count=None, v_star=u, accel=accel,
                v=torch.where(hit, u * c.boundary_damping, u), x=torch.minimum(torch.maximum(x, lo), hi))


def _eos(rho, B, rho0, gamma):
    return torch.relu(B * ((rho / rho0) ** gamma - 1.0))


def _exact_wcsph(p, x, v):
    n, h, dt, m = p.n, _f32(2.0 * p.spacing), _f32(p.dt), _f32(p.mass)
    w, gs = _cubic(h)
    near, _ = _pairs(x, x, h, p.world)
    rho = _sum(n, near, lambda i, j, r2: m * w(r2.sqrt()))
    pr = _eos(rho, _material(p, "stiffness"), 1000.0, 7.0)
    a = _non_pressure(p, near, x, v, rho, m, h)
    P = pr / (rho * rho).clamp(min=1.0e-6)
    a = a + _sum(n, near, lambda i, j, r2: (-m * (P[i] + P[j]) * gs(r2.sqrt()))[:, None] * (x[i] - x[j]), 3)
    u = v + dt * a
    x = x + dt * u
    lo, hi = _box(p)
    u = torch.where((x < lo) & (u < 0) | (x > hi) & (u > 0), u * p.config.boundary_damping, u)
    return dict(rho=rho, pressure=pr, x=torch.minimum(torch.maximum(x, lo), hi), v=u, accel=a)


def _exact_grad(p, case):
    n, h, dt, m = p.n, _f32(2.0 * p.spacing), _f32(p.dt), _f32(p.mass)
    w, gs = _cubic(h)
    lo, hi = _box(p)
    full = lambda a: torch.full((n,), _f32(a), dtype=torch.float64, device=DEV, requires_grad=True)  # noqa: E731
    ins = [p.x.double().requires_grad_(), p.v.double().requires_grad_(), full(p.attributes["stiffness"]),
           full(p.attributes["viscosity"]), full(1000.0)]
    x0, v0, B, nu, rho0 = ins
    target = (p.x + torch.tensor([0.3, 0.0, 0.0], device=DEV)).double()
    g = torch.tensor([0.0, 0.0, -10.0], dtype=torch.float64, device=DEV)

    def substep(x, v, B, nu, rho0):
        near, _ = _pairs(x.detach(), x.detach(), h)
        i, j, _ = (torch.cat(t) for t in zip(*near))
        other = i != j
        i, j = i[other], j[other]
        d = x[i] - x[j]
        r2 = (d * d).sum(1)
        r = r2.sqrt()
        zero = torch.zeros(n, dtype=torch.float64, device=DEV)
        rho = zero.index_add(0, i, m * w(r)) + m * 8.0 / (math.pi * h ** 3)
        pr = _eos(rho, B, rho0, 7.0)
        P, R = pr / (rho * rho), 1.0 / rho
        vd = ((v[i] - v[j]) * d).sum(1)
        c = (10.0 * nu[i] * m * R[j] * vd / (r2 + 0.01 * h * h) - m * (P[i] + P[j])) * gs(r)
        a = torch.zeros(n, 3, dtype=torch.float64, device=DEV).index_add(0, i, c[:, None] * d) + g
        u = v + dt * a
        x = x + dt * u
        u = torch.where((x < lo) & (u < 0) | (x > hi) & (u > 0), u * p.config.boundary_damping, u)
        return torch.minimum(torch.maximum(x, lo), hi), u
    x, v = x0, v0
    for _ in range(case["steps"]):
        x, v = torch.utils.checkpoint.checkpoint(substep, x, v, B, nu, rho0, use_reentrant=False)
    loss = ((x - target) ** 2).sum(1).mean()
    grads = torch.autograd.grad(loss, ins)
    return dict(x=x.detach(), v=v.detach(), loss=loss.detach(), grads=tuple(grads))


def _exact_separation(case, seed):
    x32, _, spacing = _column(case["n"], seed)
    x = x32.double()
    rest = _f32(2.0 * _f32(0.5 * spacing))
    margin = _f32(0.5 * spacing)
    band = max(1.5 * margin, 2.0 * margin)
    lo = torch.tensor(DEFAULT_SPEC.bound_lo, dtype=torch.float64, device=DEV).float().double()
    hi = torch.tensor(DEFAULT_SPEC.bound_hi, dtype=torch.float64, device=DEV).float().double()
    for _ in range(2):
        near, _ = _pairs(x, x, rest)

        def push(i, j, r2):
            d = r2.sqrt()
            s = torch.where((d > 1.0e-8) & (d < rest), _f32(0.55) * (rest - d) / d.clamp(min=1.0e-30),
                            torch.zeros_like(d))
            return torch.cat([s[:, None] * (x[i] - x[j]), (s > 0)[:, None].double()], 1)  # noqa: B023
        t = _sum(x.shape[0], near, push, 4)
        d = t[:, :3] / t[:, 3:].clamp(min=1.0)
        d = torch.where((x <= lo + band) & (d < 0) | (x >= hi - band) & (d > 0), torch.zeros_like(d), d)
        x = torch.minimum(torch.maximum(x + d, lo + margin), hi - margin)
    return x


def exact(case, seed):
    if case["kind"] == "grid":
        return None  # integers throughout
    if case["kind"] == "separation":
        return _exact_separation(case, seed)
    p = _problem(case, seed)
    if case["kind"] == "grad":
        return _exact_grad(p, case)
    if p.batch is not None:
        p.radius = p.batch.radius
        p.mass = p.batch.mass
    step = {"pbf": _exact_pbf, "dfsph": _exact_dfsph, "wcsph": _exact_wcsph}[p.method]
    x, v = p.x.double(), p.v.double()
    for _ in range(case.get("substeps", 1)):
        out = step(p, x, v)
        x, v = out["x"], out["v"]
    return out
