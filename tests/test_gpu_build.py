"""Grid builds one after the other in one context: every build leaves the
occupancy counts and tile sums as the next one needs them.  Sizes on both
sides of the tile-sum copies (60,000 particles), crowded cells in the block
that holds their first slot (64 particles and more, past 4,096 sorted by
digits), an empty build and non-finite positions in between; tables equal the
oracle's bit for bit."""

import numpy as np
import pytest
import torch

import oracle
from fluid_simulation_b200.newton_shim import HashGrid

pytestmark = pytest.mark.gpu
R = 0.02


def points(n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "spread":
        x = rng.uniform(-1.2, 1.2, (n, 3))
    elif kind == "columns":  # runs along z, as a lattice is numbered
        k = np.arange(n)
        x = np.stack([k // 3600, k // 60 % 60, k % 60], 1) * 0.02 + rng.uniform(0, 0.01, (n, 3))
    elif kind == "one cell":
        x = rng.uniform(0.0, R, (n, 3)) * 0.99 + R
    else:  # crowded: 50 cells of about n / 50 each
        x = rng.integers(3, 53, (n, 1)) * np.array([[R, 0.0, 0.0]]) + rng.uniform(0, R, (n, 3)) * 0.99
    return x.astype(np.float32)


@pytest.mark.parametrize("dims", [(128, 128, 128), (61, 7, 300)])
def test_builds_in_a_row_are_bit_exact(dims, cuda_device):
    g = HashGrid(*dims, device=cuda_device)
    g.reserve(130000)
    for k, (n, kind) in enumerate([(1, "spread"), (59999, "columns"), (60000, "columns"), (0, ""), (129999, "columns"),
                                   (3200, "crowded"), (3300, "crowded"), (70000, "crowded"), (4096, "one cell"),
                                   (4097, "one cell"), (512, "spread"), (130000, "spread")]):
        if n == 0:
            g.build(torch.empty(0, 3, device=cuda_device), R)
            ids, cells, starts, ends = g.tables()
            assert not starts.any() and not ends.any()
            continue
        x = points(n, kind, k)
        if kind == "spread" and n > 100:
            x[5, 1] = np.nan
            keep = np.delete(np.arange(n), 5)
        else:
            keep = np.arange(n)
        g.build(torch.as_tensor(x, device=cuda_device), R)
        ids, cells, starts, ends = (t.cpu().numpy() for t in g.tables())
        ref = oracle.grid_build(x[keep], R, dims=dims)
        m = len(keep)
        np.testing.assert_array_equal(ids[:m], keep[ref["point_ids"]])
        np.testing.assert_array_equal(cells[:m], ref["point_cells"])
        # the oracle leaves empty cells at (0, 0); here they are empty ranges
        used = ref["cell_ends"] > ref["cell_starts"]
        np.testing.assert_array_equal(starts[used], ref["cell_starts"][used])
        np.testing.assert_array_equal(ends[used], ref["cell_ends"][used])
        assert np.array_equal(starts[~used], ends[~used])
