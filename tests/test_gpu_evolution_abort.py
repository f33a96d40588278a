"""A data wait of the BSSN evolution's RK stage that gives up (k_evo_stage_bssn): the host has each CTA leave one request
out and shortens the waits."""
from __future__ import annotations

import pytest

from test_gpu_evolution_feed import varied_sim

pytestmark = pytest.mark.gpu

VISITS = 24   # fields that a stage visits with the Gamma-driver on; the update's inputs follow


@pytest.mark.parametrize("n,tree,withhold", [(8, "uniform1", 1), (8, "uniform1", VISITS + 1), (8, "uniform3", VISITS + 1),
                                             (16, "uniform1", VISITS + 1), (16, "uniform2", VISITS + 2), (32, "uniform1", 3),
                                             (32, "uniform1", VISITS + 1)])
def test_stage_that_gives_up_stores_nothing_more(am, cuda, n, tree, withhold):
    """Every CTA's request number `withhold` is left out: the error is reported once, the interiors of the fields whose
    update had not come keep their values (all of them up to the update's first request; then those past
    its first four fields at most), and a clean timestep from the same state equals that of a simulation
    that never failed, bit for bit."""
    import torch
    sim, st, fields = varied_sim(am, n, tree, 1, 3 * n)
    clean, _, _ = varied_sim(am, n, tree, 1, 3 * n)
    used, t = st["used_slots"], n + 6

    def state(s, which, f):
        return s.tensor(which, f, torch.float32)[: used * t ** 3].reshape(used, t, t, t)

    sim.set_fault_injection(spin_limit=4096, withhold_plane=withhold)
    sim.phase(am.PHASE_PREDICTOR)
    with pytest.raises(am.AmrError) as info:
        sim.synchronize()
    assert info.value.status == am.ERR_TIMEOUT
    sim.synchronize()   # reported once, then cleared
    inner = slice(3, 3 + n)
    for f in range(0 if withhold <= VISITS + 1 else 4, 24):
        start = torch.from_numpy(fields[f]).cuda().reshape(used, t, t, t)
        for which in (sim.STAGE, sim.NEW_STATE):
            assert torch.equal(state(sim, which, f)[:, inner, inner, inner], start[:, inner, inner, inner]), (which, f)
    sim.set_fault_injection(0, 0)
    for f in range(24):
        for which in (sim.OLD_STATE, sim.NEW_STATE, sim.STAGE):
            state(sim, which, f).copy_(torch.from_numpy(fields[f]).reshape(used, t, t, t))
    torch.cuda.synchronize()
    for s in (sim, clean):
        s.timestep()
        s.synchronize()
    for f in range(24):
        assert torch.equal(state(sim, sim.NEW_STATE, f), state(clean, clean.NEW_STATE, f)), f
    sim.close()
    clean.close()
