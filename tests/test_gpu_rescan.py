"""Particles whose lists overflow (192 entries; about 250 neighbours within
four spacings) rescan the grid in every later pass, over the pass's own record
of each candidate.  Inactive candidates are none of the neighbours: the step of
a model with inactive particles has, for the active ones, the bits of the step
of the active ones alone, with 16 lanes a particle and with one."""

import ctypes as C

import numpy as np
import pytest
import torch

from fluid_simulation_b200 import _lib
from fluid_simulation_b200.newton_shim import model_from_arrays
from test_gpu_lists import SP, dense_lattice
from test_gpu_scan import block, config

from fluid_simulation_b200.solver import SolverDFSPH, SolverPBF, SolverWCSPH

pytestmark = pytest.mark.gpu


def run(kind, x, v, flags, dev):
    cls = dict(wcsph=SolverWCSPH, dfsph=SolverDFSPH, pbf=SolverPBF)[kind]
    cfg, dt, attrs = config(kind, cls)
    cfg.smoothing_length_coff = 4.0
    m = model_from_arrays(x, v, 1000.0 * SP ** 3, device=dev, flags=flags, radius=0.5 * SP, attributes=attrs,
                          solver_cls=cls)
    s = cls(m, cfg)
    a, b = m.state(), m.state()
    s.step(a, b, None, None, 0.1 * dt)
    cnt = (C.c_int64 * 3)()
    _lib.check(_lib.load().fs_list_stats(m.particle_grid._ctx, cnt, 3, 1), "fs_list_stats")
    return dict(vars(b.sph), x=b.particle_q, v=b.particle_qd, accel=s._particle_accel), int(cnt[1])


@pytest.mark.parametrize("total", [2744, 40000])
@pytest.mark.parametrize("kind", ["wcsph", "dfsph", "pbf"])
def test_rescans_leave_inactive_candidates_out(kind, total, cuda_device):
    x, v = dense_lattice()
    n = len(x)
    if total > n:
        x2, v2 = block(total - n, (0.15, 0.15, 0.02), 2)
        x, v = np.concatenate([x, x2]), np.concatenate([v, v2])
    on = np.ones(total, bool)
    on[np.random.default_rng(3).choice(n, n // 12, replace=False)] = False
    both, overflowed = run(kind, x, v, on.astype(np.int32), cuda_device)
    alone, _ = run(kind, x[on], v[on], None, cuda_device)
    assert overflowed > 100
    keep = torch.as_tensor(np.nonzero(on)[0], device=cuda_device)
    for name, t in alone.items():
        assert torch.equal(both[name][keep].view(torch.int32), t.view(torch.int32)), name

