"""How many axes' ghost layers a BSSN stage writes (evo_stage_feeds, EvolveSim::stage_feeds), seen in the fill's launches
of a timestep: an axis whose every face is fed has none."""
from __future__ import annotations

import pytest

import fake_cuda


@pytest.mark.parametrize("n,depth,periodic,fills", [
    (8, 1, 1, (0, 0, 0)), (8, 1, 0, (8, 8, 8)), (8, 3, 1, (0, 0, 32)),      # small tiles; 585 domains: x and y
    (16, 1, 1, (0, 0, 0)), (16, 2, 1, (0, 0, 16)),
    (32, 1, 1, (0, 0, 0)), (32, 2, 1, (0, 0, 16)), (32, 1, 0, (8, 8, 8))])  # 32^3: z where the domains are few
def test_fill_launches_of_a_timestep(am, tmp_path, n, depth, periodic, fills):
    """Uniform trees, four fills a substep; open trees keep the launches for their outer faces."""
    out = fake_cuda.run(tmp_path, f"""
        sim = am.Sim(am.Config({n}, 3, 1.0), am.SIM_BSSN_EVOLVE, slots=sum(8 ** d for d in range({depth} + 1)), mode=am.MODE_BATCHED)
        cases.tree_uniform(sim, {depth})
        sim.set_evolution(am.Evolution(periodic={periodic}))
        fake.fake_reset(0)
        sim.timestep()
        names = [fake.fake_kernel(i).decode() for i in range(fake.fake_launches())]
        stage = {{x.split("k_evo_stage_bssn")[1][:60] for x in names if "k_evo_stage_bssn" in x}}
        print(json.dumps([[sum(f"k_evo_ghostILi{n}ELi{{a}}E" in x for x in names) for a in range(3)], sorted(stage)]))
    """)
    assert tuple(out[0]) == fills
    three = fills == (0, 0, 0)   # the kernel compiled for the axes that are fed
    assert all(("ELi3EE" in s) == three for s in out[1]), out[1]
