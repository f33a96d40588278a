"""amr_sim_autotune and the captured timestep: what it tunes on a BSSN evolution (the constraints' tiles) no timestep
launches, so the graph stays; the wave's slabs are part of its timestep, which is captured again."""
from __future__ import annotations

import pytest

import fake_cuda


@pytest.mark.parametrize("kind,captures", [("SIM_BSSN_EVOLVE", 0), ("SIM_WAVE_RK4", 1)])
def test_captures_after_tuning(am, tmp_path, kind, captures):
    out = fake_cuda.run(tmp_path, f"""
        sim = am.Sim(am.Config(16, 3, 1.0), am.{kind}, slots=9, mode=am.MODE_GRAPH)
        cases.tree_uniform(sim, 1)
        sim.timestep()
        sim.autotune(2)
        fake.fake_reset(0)
        sim.timestep()
        print(json.dumps(fake.fake_graphs()))
    """)
    assert out == captures
