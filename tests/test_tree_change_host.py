"""What a changed tree costs an evolution on the host: its lists are one per set of domains that are active together (as
many as the tree has depths), not one per substep (2^depth)."""
from __future__ import annotations

import fake_cuda


def test_uploads_after_a_tree_change(am, tmp_path):
    """The bytes that the next call uploads: the octree's arrays, the feed table and, per set, at most two lists of
    domains and twice six faces a domain."""
    out = fake_cuda.run(tmp_path, """
        slots = 1600
        sim = am.Sim(am.Config(8, 3, 1.0), am.SIM_BSSN_EVOLVE, slots=slots, mode=am.MODE_GRAPH)
        cases.tree_random(sim, 6, .3, 3)
        sim.timestep()
        st = sim.state()
        out = {"slots": slots, "used": int(st["used_slots"]), "depth": int(st["max_depth"])}
        for name, call in (("norms", sim.constraint_norms), ("timestep", sim.timestep)):
            sim.set_octree(st)
            fake.fake_reset(0)
            call()
            out[name] = fake.fake_uploaded()
        print(json.dumps(out))
    """)
    assert out["depth"] == 6
    sets = out["depth"] + 1
    most = out["slots"] * (4 + 32 + 48 + 1 + 24) + 4 * out["used"] * (2 * sets + 2 + 2 * 6 * sets)
    assert out["norms"] <= most and out["timestep"] <= most, (out, most)


def test_nothing_is_listed_after_tuning(am, tmp_path):
    """amr_sim_autotune lists what the timesteps that follow need: the first of them uploads nothing."""
    out = fake_cuda.run(tmp_path, """
        out = []
        for kind in (am.SIM_BSSN_EVOLVE, am.SIM_WAVE_RK4):
            sim = am.Sim(am.Config(16, 3, 1.0), kind, slots=64, mode=am.MODE_GRAPH)
            cases.tree_uneven(sim)
            sim.autotune(2)
            fake.fake_reset(0)
            sim.timestep()
            out.append(fake.fake_uploaded())
        print(json.dumps(out))
    """)
    assert out == [0, 0]
