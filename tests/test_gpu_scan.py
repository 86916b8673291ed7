"""The grid scan at the edges of its tiles: groups of four slots, pieces of 32
candidates, 12 pieces between two visits, lists of 192 entries; inactive
candidates, rows that wrap, dims that are no power of two.

Densities against a float64 sum over all pairs: k positive FP32 terms, each a
few ulp off, summed one after the other, are within (k + 16) 2^-23 of it
(relative).  DFSPH's neighbour counts (candidates, no distance test) equal the
oracle's candidate lists.

Small scenes give several lanes to a particle (16, 8, 4 or 1 by the particle
count): a scene stepped together with particles far away from it, whose number
moves the count across those limits, keeps every bit of its step alone."""

import numpy as np
import pytest
import torch

import oracle
from fluid_simulation_b200.newton_shim import HashGrid, model_from_arrays
from fluid_simulation_b200.solver import SolverDFSPH, SolverPBF, SolverWCSPH

pytestmark = pytest.mark.gpu
SP = 0.01
H = 2 * SP


def cloud(n, centre, seed):
    """n points around `centre`, half of them within one cell, the others over 5 h."""
    rng = np.random.default_rng(seed)
    near = rng.uniform(0.0, 1.0, (n - n // 2, 3)) * H
    wide = rng.uniform(-2.5, 2.5, (n // 2, 3)) * H
    x = np.concatenate([near, wide]) + np.asarray(centre)
    return x.astype(np.float32)[rng.permutation(n)]


def step(cls, x, flags, dims, dev, dt):
    n = len(x)
    attrs = dict(particle_mask=0, rest_density=1000.0, surface_tension=0.0, viscosity=0.0)
    if cls is SolverWCSPH:
        attrs.update(stiffness=1.0, exponent=1.0)
    m = model_from_arrays(x, np.zeros_like(x), 1000.0 * SP ** 3, device=dev, flags=flags, radius=0.5 * SP,
                          attributes=attrs, solver_cls=cls)
    m.particle_grid = HashGrid(*dims, device=dev)
    m.particle_grid.reserve(n)
    solver = cls(m, cls.SphConfig(particle_radius=0.5 * SP, particle_length=SP, smoothing_length_coff=2.0,
                                  bound_width=1e4, bound_height=1e4, bound_length=1e4))
    a, b = m.state(), m.state()
    solver.step(a, b, None, None, dt)
    torch.cuda.synchronize()
    return b


def density64(x, active):
    d = np.linalg.norm(x[:, None].astype(np.float64) - x[None].astype(np.float64), axis=2) / np.float64(np.float32(H))
    k = 8.0 / (np.pi * H ** 3)
    w = np.where(d <= 0.5, k * (6 * d ** 3 - 6 * d ** 2 + 1), 2 * k * np.clip(1 - d, 0, None) ** 3)
    w = np.where((d <= 1.0) & active[None], w, 0.0)
    return np.where(active, 1000.0 * SP ** 3 * w.sum(1), 0.0), int((w > 0).sum(1).max())


@pytest.mark.parametrize("dims", [(128, 128, 128), (7, 5, 3)])
@pytest.mark.parametrize("centre", [(0.31, 0.27, 0.2), (0.0, 0.0, 0.0)])
@pytest.mark.parametrize("n", [2, 3, 5, 31, 64, 65, 129, 500, 2000])
def test_scan_edges(n, centre, dims, cuda_device):
    x = cloud(n, centre, n)
    flags = np.ones(n, np.int32)
    flags[::7] = 0
    if n < 7:
        flags[:] = 1
    active = flags == 1
    want, hits = density64(x, active)
    got = step(SolverWCSPH, x, flags, dims, cuda_device, 1e-9).sph.rho.cpu().numpy()
    err = np.abs(got - want).max() / max(want.max(), 1e-30)
    assert err <= (hits + 16) * 2.0 ** -23, (err, hits)
    off, cand = oracle.grid_candidates(x, np.float32(H), dims=dims)
    count = np.array([np.count_nonzero(active[c] & (c != i)) for i, c in
                      enumerate(np.split(np.asarray(cand), np.asarray(off)[1:-1]))])
    got = step(SolverDFSPH, x, flags, dims, cuda_device, 1e-9).sph.neighbor_count.cpu().numpy()
    assert np.array_equal(got, np.where(active, count, 0))


def block(n, corner, seed):
    """n particles of a jittered lattice at rest spacing, moving."""
    side = int(np.ceil(n ** (1.0 / 3.0)))
    k = np.arange(n)
    g = np.stack([k // side ** 2, k // side % side, k % side], 1)
    rng = np.random.default_rng(seed)
    x = (g + rng.uniform(-0.2, 0.2, g.shape)) * SP + np.asarray(corner)
    return x.astype(np.float32), rng.normal(0.0, 0.1, x.shape).astype(np.float32)


def config(kind, cls):
    """Config, time step and model attributes with every pass at work; DFSPH never ends early (its residual is a mean
    over all particles)."""
    base = dict(particle_radius=0.5 * SP, particle_length=SP, smoothing_length_coff=2.0, bound_width=0.6,
                bound_height=0.6, bound_length=0.5, boundary_damping=0.0)
    attrs = dict(particle_mask=0, rest_density=1000.0, surface_tension=0.01, viscosity=0.005)
    if kind == "wcsph":
        attrs.update(stiffness=2.5e5, exponent=7.0)
        return cls.SphConfig(**base), 1e-4, attrs
    if kind == "dfsph":
        return cls.SphConfig(max_rho_iterations=3, max_vel_iterations=4, warm_start=False, eta_density=-1.0,
                             eta_divergence=-1.0, **base), 1e-3, attrs
    return cls.PbfConfig(max_iterations=3, lambda_epsilon=100.0, max_delta_position=0.25 * SP, xsph_c=0.05,
                         scorr_k=1e-4, **base), 1e-3, attrs


def run_step(kind, x, v, mass, dev):
    cls = dict(wcsph=SolverWCSPH, dfsph=SolverDFSPH, pbf=SolverPBF)[kind]
    cfg, dt, attrs = config(kind, cls)
    m = model_from_arrays(x, v, mass, device=dev, radius=0.5 * SP, attributes=attrs, solver_cls=cls)
    s = cls(m, cfg)
    a, b = m.state(), m.state()
    s.step(a, b, None, None, dt)
    return dict(vars(b.sph), x=b.particle_q, v=b.particle_qd, accel=s._particle_accel)


@pytest.mark.parametrize("n", [3000, 40000])
@pytest.mark.parametrize("kind", ["wcsph", "dfsph", "pbf"])
def test_particles_of_another_mass_far_away_change_no_bit(kind, n, cuda_device):
    """One mass for all is not loaded for each neighbour; one far particle of another mass has them all loaded."""
    x, v = block(n, (-0.55, -0.55, 0.02), 1)
    far = np.array([[0.55, 0.55, 0.9]], np.float32)
    mass = 1000.0 * SP ** 3
    same = run_step(kind, np.concatenate([x, far]), np.concatenate([v, 0 * far]), mass, cuda_device)
    masses = np.full(n + 1, mass, np.float32)
    masses[n] *= 2.0
    mixed = run_step(kind, np.concatenate([x, far]), np.concatenate([v, 0 * far]), masses, cuda_device)
    for name, t in same.items():
        assert torch.equal(t[:n], mixed[name][:n]), name


@pytest.mark.parametrize("total", [4999, 6000, 6001, 14000, 14001, 38000, 38001])
@pytest.mark.parametrize("kind", ["wcsph", "dfsph", "pbf"])
@pytest.mark.parametrize("corners", [((-0.55, -0.55, 0.02), (-0.2, -0.2, 0.02)),
                                     ((-0.07, -0.07, 0.02), (0.15, 0.15, 0.02))])  # around x = y = 0: wide rows, wraps
def test_lanes_per_particle_change_no_bit(kind, total, corners, cuda_device):
    n = 2500
    x, v = block(n, corners[0], 1)
    x2, v2 = block(total - n, corners[1], 2)

    mass = 1000.0 * SP ** 3
    alone = run_step(kind, x, v, mass, cuda_device)
    both = run_step(kind, np.concatenate([x, x2]), np.concatenate([v, v2]), mass, cuda_device)
    for name, t in alone.items():
        assert torch.equal(t, both[name][:n]), name


@pytest.mark.parametrize("m", [2, 4, 5, 188, 189, 190, 191, 192, 193, 194, 197])
@pytest.mark.parametrize("kind", ["wcsph", "dfsph", "pbf"])
def test_full_lists_of_one_lane_change_no_bit(kind, m, cuda_device):
    """m particles that all see each other, around the 192 entries a list holds (the particle itself counts), alone
    with 16 lanes each and with so many others that each has one."""
    rng = np.random.default_rng(m)
    d = rng.normal(size=(m, 3))
    r = 0.45 * H * rng.uniform(0.0, 1.0, (m, 1)) ** (1.0 / 3.0)
    x = (d / np.linalg.norm(d, axis=1, keepdims=True) * r + (-0.45, -0.45, 0.2)).astype(np.float32)
    v = rng.normal(0.0, 0.1, x.shape).astype(np.float32)
    x2, v2 = block(38100, (-0.07, -0.07, 0.02), 2)
    mass = 1000.0 * SP ** 3
    alone = run_step(kind, x, v, mass, cuda_device)
    both = run_step(kind, np.concatenate([x, x2]), np.concatenate([v, v2]), mass, cuda_device)
    for name, t in alone.items():
        assert torch.equal(t.view(torch.int32), both[name][:m].view(torch.int32)), name
