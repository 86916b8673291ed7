"""The launch autotuner's candidates where several lanes share a particle (no GPU): particles per thread has no effect
there, so that its values are not timed against each other."""

import pytest

from fluid_simulation_b200 import _lib
from fluid_simulation_b200.autotune import DEFAULT, Tuning, autotune, candidates


@pytest.mark.parametrize("kind,ratios", [("pbf", 1), ("dfsph", 1), ("wcsph", 2)])
def test_particles_per_thread_is_tuned_with_one_lane_only(kind, ratios):
    assert candidates(kind) == candidates(kind, lanes=1)
    for lanes in (4, 8, 16):
        c = candidates(kind, lanes=lanes)
        assert c[0] == Tuning(*DEFAULT) and len(c) == len(set(c)) == 3 * ratios
        assert all(t.particles_per_thread == 1 for t in c)


@pytest.mark.parametrize("n,timed", [(1, 3), (38000, 3), (38001, 9), (4194304, 9)])
def test_autotune_times_what_differs(n, timed, monkeypatch):
    class SolverPBF:
        class model:
            particle_count = n

            class particle_grid:
                _ctx = None
    monkeypatch.setattr("fluid_simulation_b200.autotune.set_tuning", lambda ctx, t: None)
    times = autotune(SolverPBF(), None, 1e-3, timer=lambda t: 1.0)["times_ms"]
    assert len(times) == timed


def test_lanes_per_particle():
    lanes = _lib.load().fs_lanes_per_particle
    assert [lanes(n) for n in (1, 6000, 6001, 14000, 14001, 38000, 38001)] == [16, 16, 8, 8, 4, 4, 1]
