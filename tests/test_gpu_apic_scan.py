"""Particle separation where its scan changes: 24 and more candidates within
reach of a particle, queries that wrap modulo the grid's dims, few cells;
bit-for-bit equal to the oracle."""

import numpy as np
import pytest
import torch

import oracle
from fluid_simulation_b200.apic import ParticleSeparation
from fluid_simulation_b200.newton_shim import model_from_arrays

pytestmark = pytest.mark.gpu
R = 0.01


@pytest.mark.parametrize("lo", [(-0.3, -0.2, 0.0), (0.15, 0.05, 0.1)])  # cells of both signs: rows that wrap, or none
@pytest.mark.parametrize("cluster", [2, 23, 24, 25, 26, 200])
def test_clusters_match_the_oracle(cluster, lo, cuda_device):
    rng = np.random.default_rng(cluster)
    hi = tuple(a + b for a, b in zip(lo, (0.37, 0.11, 0.05)))
    spread = rng.uniform(lo, hi, (3000, 3))
    centres = spread[:40]
    x = np.concatenate([spread] + [c + rng.uniform(-0.3, 0.3, (cluster, 3)) * R for c in centres])
    x = np.clip(x, lo, hi).astype(np.float32)[rng.permutation(3000 + 40 * cluster)]
    flags = np.ones(len(x), np.int32)
    flags[::11] = 0
    m = model_from_arrays(x, np.zeros_like(x), 1.0, device=cuda_device, flags=flags, radius=0.5 * R)
    sep = ParticleSeparation(m, ParticleSeparation.Config(bound_lo=lo, bound_hi=hi))
    st = m.state()
    sep.apply(st)
    want, push = oracle.apic_separation(x, flags, sep.parameters(), "f32")
    assert np.array_equal(st.particle_q.cpu().numpy(), want)
    assert np.array_equal(sep._sep_delta.cpu().numpy(), push)
    assert torch.isfinite(st.particle_q).all()
