"""The grid scan at its edges for every number of lanes a particle can have
(8, 4 or 1 above 6,000, 14,000 and 38,000 particles): a cloud beside so many
particles far away that the count takes each of them.  Inactive candidates,
dims that are no power of two and alias the cloud with the far particles (rows
of more than 12 pieces, resumed in the middle of a row; rows that wrap), and
queries below the shifted range of cells (a segment per cell, cells met more
than once).

Densities against a float64 sum over the oracle's candidates: k positive FP32
terms, each a few ulp off, summed one after the other, are within (k + 16)
2^-23 of it (relative).  DFSPH's neighbour counts equal those candidates."""

import numpy as np
import pytest

import oracle
from fluid_simulation_b200.solver import SolverDFSPH, SolverWCSPH
from test_gpu_scan import H, SP, cloud, step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [7000, 20000, 40000])
@pytest.mark.parametrize("dims", [(128, 128, 128), (7, 5, 3), (61, 7, 300)])
@pytest.mark.parametrize("centre", [(0.31, 0.27, 0.2), (0.0, 0.0, 0.0), (-22000.0, 0.27, 0.2)])
def test_scan_edges_beside_many_particles(total, dims, centre, cuda_device):
    n = 500
    rng = np.random.default_rng(total)
    far = rng.uniform(-0.3, 0.3, (total - n, 3)) + np.asarray(centre) + np.array([2.0, 2.0, 2.0])
    x = np.concatenate([cloud(n, centre, n), far.astype(np.float32)])
    flags = np.ones(total, np.int32)
    flags[::7] = 0
    active = flags == 1
    off, cand = oracle.grid_candidates(x, np.float32(H), x[:n], np.float32(H), dims=dims)
    cand, off = np.asarray(cand), np.asarray(off)
    i = np.repeat(np.arange(n), np.diff(off))
    d = np.linalg.norm(x[i].astype(np.float64) - x[cand].astype(np.float64), axis=1) / np.float64(np.float32(H))
    k = 8.0 / (np.pi * H ** 3)
    w = np.where(d <= 0.5, k * (6 * d ** 3 - 6 * d ** 2 + 1), 2 * k * np.clip(1 - d, 0, None) ** 3)
    w = np.where((d <= 1.0) & active[cand], w, 0.0)
    rho = np.where(active[:n], 1000.0 * SP ** 3 * np.bincount(i, w, n), 0.0)
    hits = int(np.bincount(i, w > 0, n).max())
    got = step(SolverWCSPH, x, flags, dims, cuda_device, 1e-9).sph.rho.cpu().numpy()[:n]
    err = np.abs(got - rho).max() / rho.max()
    assert err <= (hits + 16) * 2.0 ** -23, (err, hits)
    count = np.bincount(i, active[cand] & (cand != i), n)
    got = step(SolverDFSPH, x, flags, dims, cuda_device, 1e-9).sph.neighbor_count.cpu().numpy()[:n]
    assert np.array_equal(got, np.where(active[:n], count, 0))
