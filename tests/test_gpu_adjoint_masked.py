"""Gradients of the WCSPH adjoint beside particles that do not move: masked
ones (with mass, and with none: the mass is the divisor of the cohesion term,
which a particle that does not move has no use for), inactive ones, and
unequal masses, at every number of lanes a particle can have (16, 8, 4, 1 by
the particle count; particles far away make up the count).  One substep
against FP64 tape gradients of the same step; 1e-3 norm-relative, the
tolerance of the other gradient tests."""

import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

import wcsph_tape
from adjoint_util import CFG, DT, GRAVITY, MASS, SPACING, block, params
from fluid_simulation_b200.diff import DiffWCSPH
from fluid_simulation_b200.newton_shim import model_from_arrays
from fluid_simulation_b200.solver import SolverWCSPH
from golden_io import rel_err

pytestmark = pytest.mark.gpu
GTOL = 1e-3
NAMES = ("x0", "v0", "stiffness", "viscosity", "rest_density")


def scene(total):
    """A compressed block at the floor and the -x wall, every fifth particle masked (every other one of those without
    mass), every seventh of the others inactive, masses 80 to 120 %; and total - 9^3 particles at rest far away."""
    x, v = block(side=9, seed=3)
    n = len(x)
    k = np.arange(n)
    mask = (k % 5 == 0).astype(np.int32)
    flags = np.where((k % 7 == 3) & (mask == 0), 0, 1).astype(np.int32)
    mass = (MASS * np.random.default_rng(5).uniform(0.8, 1.2, n)).astype(np.float32)
    mass[k % 10 == 0] = 0.0
    m = total - n
    side = int(np.ceil(m ** (1.0 / 3.0)))
    j = np.arange(m)
    far = (np.stack([j // side ** 2, j // side % side, j % side], 1) * 3.0 * SPACING + 2.0).astype(np.float32)
    cat = np.concatenate
    return (n, cat([x, far]), cat([v, np.zeros_like(far)]), cat([mask, np.zeros(m, np.int32)]),
            cat([flags, np.ones(m, np.int32)]), cat([mass, np.full(m, MASS, np.float32)]))


def tape_step(x, v, mass, mask, flags, prm, cfg):
    """One substep in FP64 (wcsph_tape.substep with particles that do not move or take no part)."""
    n = x.shape[0]
    h = cfg["smoothing_length_coff"] * cfg["particle_length"]
    active = torch.as_tensor(flags == 1)
    dyn = active & torch.as_tensor(mask == 0)
    pairs = cKDTree(x.detach().numpy()).query_pairs(h, output_type="ndarray")
    i = torch.as_tensor(np.concatenate([pairs[:, 0], pairs[:, 1]]), dtype=torch.long)
    j = torch.as_tensor(np.concatenate([pairs[:, 1], pairs[:, 0]]), dtype=torch.long)
    i, j = i[active[i] & active[j]], j[active[i] & active[j]]
    mv = prm["rest_density"] * (mass / prm["rest_density"].clamp(min=1e-6))
    zero = torch.zeros(n, dtype=torch.float64)
    d = x[i] - x[j]
    r = torch.sqrt((d * d).sum(1))
    rho = mv * wcsph_tape.cubic_w(zero, h) + zero.index_add(0, i, mv[j] * wcsph_tape.cubic_w(r, h))
    p = torch.relu(prm["stiffness"] * ((rho / prm["rest_density"].clamp(min=1e-6)) ** prm["exponent"] - 1.0))
    P, R = p / (rho * rho).clamp(min=1e-6), 1.0 / rho.clamp(min=1e-6)
    moves = dyn[i]
    i, j, d, r = i[moves], j[moves], d[moves], r[moves]
    gs = wcsph_tape.cubic_gs(r, h)
    visc = 10.0 * prm["viscosity"][i] * mass[j] * R[j] * ((v[i] - v[j]) * d).sum(1) / (r * r + 0.01 * h * h)
    wc = (prm["surface_tension"][i] / mass[i]) * mass[j] * wcsph_tape.cubic_w(r.clamp(min=cfg["particle_radius"]), h)
    c = (visc - mass[j] * (P[i] + P[j])) * gs - wc
    a = torch.zeros(n, 3, dtype=torch.float64).index_add(0, i, c[:, None] * d) + torch.tensor(GRAVITY).double()
    v1 = v + DT * a
    x1, v1 = wcsph_tape.walls(x + DT * v1, v1, cfg["bound_width"], cfg["bound_height"], cfg["bound_length"],
                              cfg["boundary_damping"])
    return torch.where(dyn[:, None], x1, x), torch.where(dyn[:, None], v1, v)


@pytest.mark.parametrize("total", [1000, 7000, 20000, 40000])
def test_gradients_beside_particles_that_do_not_move(total, cuda_device):
    n, x, v, mask, flags, mass = scene(total)
    cfg = dict(CFG, bound_width=CFG["bound_width"], bound_height=10.0, bound_length=10.0)
    prm = params(total, seed=4)
    rng = np.random.default_rng(6)
    wx, wv = rng.normal(size=(total, 3)), rng.normal(size=(total, 3))
    wx[n:] = wv[n:] = 0.0  # the far particles lie behind the +x wall: their own gradients are not looked at

    m = model_from_arrays(x, v, mass, device=cuda_device, flags=flags, radius=cfg["particle_radius"],
                          gravity=(GRAVITY,), attributes=dict(prm, particle_mask=mask), solver_cls=SolverWCSPH)
    sim = DiffWCSPH(m, SolverWCSPH.SphConfig(**cfg), DT, checkpoint_every=1)
    leaves = [torch.tensor(a, device=cuda_device, requires_grad=True)
              for a in (x, v, prm["stiffness"], prm["viscosity"], prm["rest_density"])]
    xT, vT = sim.rollout(*leaves, 1)
    assert torch.isfinite(xT).all() and torch.isfinite(vT).all()
    ((xT * torch.as_tensor(wx, device=cuda_device)).sum()
     + 1e-3 * (vT * torch.as_tensor(wv, device=cuda_device)).sum()).backward()
    got = [t.grad.double().cpu().numpy()[:n] for t in leaves]

    tl = [torch.tensor(a[:n], dtype=torch.float64, requires_grad=True)
          for a in (x, v, prm["stiffness"], prm["viscosity"], prm["rest_density"])]
    tp = dict(stiffness=tl[2], viscosity=tl[3], rest_density=tl[4],
              exponent=torch.tensor(prm["exponent"][:n]).double(),
              surface_tension=torch.tensor(prm["surface_tension"][:n]).double())
    xr, vr = tape_step(tl[0], tl[1], torch.tensor(mass[:n]).double(), mask[:n], flags[:n], tp, cfg)
    ((xr * torch.as_tensor(wx[:n])).sum() + 1e-3 * (vr * torch.as_tensor(wv[:n])).sum()).backward()
    want = [t.grad.numpy() for t in tl]
    assert all(np.isfinite(w).all() for w in want)
    errs = {nm: rel_err(g, w) for nm, g, w in zip(NAMES, got, want)}
    print(errs)
    assert all(e <= GTOL for e in errs.values()), errs
    assert all(np.abs(w).max() > 0 for w in want)
