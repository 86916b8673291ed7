"""Particles whose lists overflow (192 entries; about 250 neighbours within
four spacings) rescan the grid in every later pass, over the pass's own record
of each candidate.  Inactive candidates are none of the neighbours: the step of
a model with inactive particles has, for the active ones, the bits of the step
of the active ones alone, with 16 lanes a particle and with one.  The passes
that run by themselves scan the grid the same way."""

import ctypes as C

import numpy as np
import pytest
import torch

from fluid_simulation_b200 import _lib
from fluid_simulation_b200.newton_shim import HashGrid, model_from_arrays
from fluid_simulation_b200.solver import SolverDFSPH, SolverPBF, SolverWCSPH
from fluid_simulation_b200.solver import _common as cm
from test_gpu_lists import SP, dense_lattice
from test_gpu_scan import block, config

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



def passes(x, v, flags, lam, dev):
    """DFSPH's rate and correction and PBF's delta by themselves."""
    n = len(x)
    attrs = dict(particle_mask=0, rest_density=1000.0, surface_tension=0.0, viscosity=0.0)
    m = model_from_arrays(x, v, 1000.0 * SP ** 3, device=dev, flags=flags, radius=0.5 * SP, attributes=attrs,
                          solver_cls=SolverPBF)
    h = 2.0 * SP
    m.particle_grid = HashGrid(device=dev)
    m.particle_grid.build(m.particle_q, h)
    ctx, ms, lib = m.particle_grid._ctx, cm.model_struct(m), _lib.load()
    st = torch.cuda.current_stream(dev).cuda_stream
    p = SolverPBF(m, SolverPBF.PbfConfig(particle_radius=0.5 * SP, particle_length=SP, smoothing_length_coff=2.0,
                                         scorr_k=1e-4)).params(1e-3)
    f = torch.as_tensor(lam, device=dev)
    rho = 1000.0 + f
    rate, dp, vs = torch.empty(n, device=dev), torch.empty(n, 3, device=dev), m.particle_qd.clone()
    _lib.check(lib.fs_dfsph_divergence(ctx, C.byref(ms), m.particle_q.data_ptr(), m.particle_qd.data_ptr(), h,
                                       rate.data_ptr(), st), "divergence")
    _lib.check(lib.fs_dfsph_correct(ctx, C.byref(ms), m.particle_q.data_ptr(), vs.data_ptr(), rho.data_ptr(),
                                    f.data_ptr(), h, 1e-3, st), "correct")
    _lib.check(lib.fs_pbf_delta(ctx, C.byref(ms), m.particle_q.data_ptr(), f.data_ptr(), C.byref(p), dp.data_ptr(), st),
               "delta")
    return dict(rate=rate, v_star=vs, delta=dp)


@pytest.mark.parametrize("total", [2744, 40000])
def test_passes_by_themselves_leave_inactive_candidates_out(total, cuda_device):
    x, v = dense_lattice()
    n = len(x)
    if total > n:
        x2, v2 = block(total - n, (0.15, 0.15, 0.02), 2)
        x, v = np.concatenate([x, x2]), np.concatenate([v, v2])
    rng = np.random.default_rng(4)
    on = np.ones(total, bool)
    on[rng.choice(n, n // 12, replace=False)] = False
    lam = rng.uniform(0.0, 1e-3, total).astype(np.float32)
    both = passes(x, v, on.astype(np.int32), lam, cuda_device)
    alone = passes(x[on], v[on], None, lam[on], cuda_device)
    keep = torch.as_tensor(np.nonzero(on)[0], device=cuda_device)
    for name, t in alone.items():
        assert float(t.abs().max()) > 0.0
        assert torch.equal(both[name][keep].view(torch.int32), t.view(torch.int32)), name
