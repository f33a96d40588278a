"""The SimpleWave plugin's triage on given criterion values, on the CPU (no kernel runs; the criterion's buffer is
written by the test)."""
from __future__ import annotations

import fake_cuda


def test_no_domain_is_added_to_one_that_was_removed(am, tmp_path):
    """A calm depth-2 domain whose lifetime counts is removed with its children; the children's own octants ask for
    refinement.  Nothing may be added to them: a position is none or lies under its parent's."""
    out = fake_cuda.run(tmp_path, """
        n, h, q = 28, 14, 7
        sim = am.Sim(am.Config(n, 2, 100.0), am.SIM_WAVE, slots=32, mode=am.MODE_BATCHED)
        for p in (0, 1, 9):
            for c in range(8):
                sim.add_node(p, c)
        st = sim.state()
        assert st["used_slots"] == 25 and st["max_depth"] == 3
        st["lifetime"] = st["lifetime"].copy()
        st["lifetime"][9] = 20
        sim.set_octree(st)
        octants = np.ones((25, 8), np.float32)
        octants[9] = 0
        octants[17:, 0] = 50
        crit = np.zeros((25, n * n), np.float32)
        for o, at in enumerate((0, h, n * q, h + n * q, n * h, h + n * h, n * q + n * h, h + n * q + n * h)):
            crit[:, at] = octants[:, o]
        ptr, count = sim.buffer(sim.WAVE_CRIT, 0)
        ctypes.memmove(ptr, crit.ctypes.data, crit.nbytes)
        sim.phase(am.PHASE_MODIFY_NODES)
        st = sim.state()
        print(json.dumps([int(st["used_slots"]), int(st["max_depth"]), [int(p) for p in st["positions"][:25]], [int(p) for p in st["parent"][:25]]]))
    """)
    used, depth, positions, parents = out
    assert (used, depth) == (17, 2)
    free = 0xFFFFFFFF
    for i, p in enumerate(positions[1:], 1):
        assert p == free or (positions[parents[i]] != free and p >> 27 == (positions[parents[i]] >> 27) + 1), (i, hex(p))
    assert positions[9] == free and positions[17:] == [free] * 8
