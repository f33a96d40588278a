"""What a changed tree costs an evolution on the host: its lists are one per set of domains that are active together (as
many as the tree has depths), not one per substep (2^depth)."""
from __future__ import annotations

import pytest

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


@pytest.mark.parametrize("call", ["autotune", "constraint_norms", "timestep"])
def test_one_call_lists_for_all(am, tmp_path, call):
    """What a first call lists (it synchronises) serves the timesteps that follow, which upload nothing: a caller may
    capture them into a graph of its own."""
    out = fake_cuda.run(tmp_path, f"""
        out = []
        for kind in (am.SIM_BSSN_EVOLVE, am.SIM_WAVE_RK4):
            if kind == am.SIM_WAVE_RK4 and {call!r} == "constraint_norms":
                continue
            sim = am.Sim(am.Config(16, 3, 1.0), kind, slots=64, mode=am.MODE_BATCHED)
            cases.tree_uneven(sim)
            sim.{call}()
            fake.fake_reset(0)
            sim.timestep()
            out.append(fake.fake_uploaded())
        print(json.dumps(out))
    """)
    assert out and not any(out), out
