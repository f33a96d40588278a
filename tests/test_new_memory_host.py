"""New device memory is zeroed by cudaMemset, on the legacy stream, which a simulation's (non-blocking) stream does not
wait for: where other work holds the GPU, the zeros can land after what the simulation has written there since.
No call may return with such a write still queued for memory that the simulation uses."""
from __future__ import annotations

import fake_cuda


def test_no_zeroing_is_queued_when_a_call_returns(am, tmp_path):
    out = fake_cuda.run(tmp_path, """
        out = {}
        def check(what): out[what] = fake.fake_queued()
        for name, kind, cfg, mode in (("bssn", am.SIM_BSSN, (16, 3, 1.0), am.MODE_GRAPH), ("wave", am.SIM_WAVE, (28, 2, 1.0), am.MODE_BATCHED),
                                      ("rk4", am.SIM_WAVE_RK4, (16, 3, 1.0), am.MODE_GRAPH), ("evolve", am.SIM_BSSN_EVOLVE, (8, 3, 1.0), am.MODE_GRAPH)):
            sim = am.Sim(am.Config(*cfg), kind, slots=64, mode=mode)
            check(name + " created")
            cases.tree_uneven(sim)
            sim.timestep()
            check(name + " first timestep")
            sim.add_nodes([2] * 8, list(range(8)))   # longer lists
            sim.timestep()
            check(name + " timestep of a larger tree")
            if kind == am.SIM_BSSN_EVOLVE:
                n = ctypes.c_uint32()
                assert am.load().amr_sim_tile_features(sim.h, None, None, None, 0, ctypes.byref(n)) == 5
                sim.regrid(am.Regrid())
                check(name + " regrid")
        print(json.dumps(out))
    """)
    assert out and all(v == 0 for v in out.values()), out


def test_a_loaded_checkpoint_has_arrived(am, tmp_path):
    """cudaMemcpy from pageable memory may return before the last bytes reach the device, on the legacy stream too."""
    (tmp_path / "at").mkdir()
    out = fake_cuda.run(tmp_path, f"""
        sim = am.Sim(am.Config(8, 3, 1.0), am.SIM_BSSN_EVOLVE, slots=9, mode=am.MODE_BATCHED)
        sim.save_checkpoint({str(tmp_path / "at")!r})
        sim.load_checkpoint({str(tmp_path / "at")!r})
        print(json.dumps(fake.fake_queued()))
    """)
    assert out == 0
