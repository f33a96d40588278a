"""The SimpleWave plugin's timestep where its triage takes the deepest levels away between substeps, so that domains
become active which the substep's restriction did not cover: the ghost fill must not take their old field for
their new one."""
from __future__ import annotations

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

PHASES = ("COPY_BACK", "MODIFY_NODES", "PREDICTOR", "COPY_BOUNDS", "CORRECTOR", "INCREMENT_TIMER")


def wave_sim(am):
    """Root, 8 children, 8 grandchildren in child 0, one depth-3 domain in the first of those with 8 children.  The
    depth-4 domains hold a checkerboard (large second differences, mean .5), so that at substep 2 of 16, when
    depths 3 and 4 alone are active, the triage removes their smooth parent, whose lifetime counts, and them with
    it.  The counter is then 0 of 4, and every domain left is active."""
    import torch
    cfg = am.Config(28, 2, 100.0)
    n, t = cfg.size_domain, cfg.total
    sim = am.Sim(cfg, am.SIM_WAVE, slots=27, mode=am.MODE_BATCHED)
    for c in range(8):
        sim.add_node(0, c)
    first = int(sim.state()["children"][0])
    for c in range(8):
        sim.add_node(first, c)
    second = int(sim.state()["children"][first * 8])
    sim.add_node(second, 0)
    third = int(sim.state()["children"][second * 8])
    for c in range(8):
        sim.add_node(third, c)
    sim.synchronize()
    st = sim.state()
    used = st["used_slots"]
    assert used == 26 and st["max_depth"] == 4
    st["lifetime"] = st["lifetime"].copy()
    st["lifetime"][third] = 20
    sim.set_octree(st)
    xyz = cases.cell_coordinates(st["positions"], used, n, 2, 100.0)
    f = (.5 + .2 * cases.smooth_field(xyz, 100.0, 0, 5, noise=0.0)).astype(np.float32).reshape(used, t, t, t)
    sign = (-1.0) ** np.indices((t, t, t)).sum(0)
    for c in range(8):
        f[int(st["children"][third * 8 + c])] = (.5 + .3 * sign).astype(np.float32)
    f[third] = .5
    for which in (am.Sim.OLD, am.Sim.NEW):
        sim.tensor(which)[: used * t ** 3].copy_(torch.from_numpy(f.reshape(-1)).cuda())
    torch.cuda.synchronize()
    return sim, first


def test_fill_after_the_deepest_levels_are_removed(am, cuda):
    """One timestep against the same phases called one by one (whose ghost fill stages every value): both fields,
    ghosts included, and the tree bit for bit."""
    whole, _ = wave_sim(am)
    phased, first = wave_sim(am)
    whole.timestep()
    seen = []
    while True:
        for ph in PHASES:
            before = phased.state()
            phased.phase(getattr(am, "PHASE_" + ph))
            after = phased.state()
            if ph == "MODIFY_NODES" and after["max_depth"] != before["max_depth"]:
                seen.append((before["max_depth"], before["timer"], after["max_depth"], after["timer"]))
        if phased.state()["timer"] == 0:
            break
    assert seen[0] == (4, 2, 2, 0)   # the case is the one described above
    whole.synchronize()
    phased.synchronize()
    a, b = whole.state(), phased.state()
    assert all(np.array_equal(a[k], b[k]) for k in a)
    assert int(a["children"][first * 8]) != -1   # depth-2 domains beside depth-1 ones are left
    cells = a["used_slots"] * whole.cfg.total ** 3
    for which in (am.Sim.NEW, am.Sim.OLD):
        x = whole.tensor(which)[:cells].cpu().numpy().view(np.uint32)
        y = phased.tensor(which)[:cells].cpu().numpy().view(np.uint32)
        assert np.count_nonzero(x != y) == 0, f"buffer {which}: {np.count_nonzero(x != y)} of {cells} words differ"
    whole.close()
    phased.close()


def test_fill_with_slots_that_hold_no_domain(am, cuda):
    """Slots whose domain was removed keep their boundary records, and the fill follows them though no restriction covered
    their sources: one timestep against the phases called one by one, every word of the used slots bit for bit."""
    import torch
    cfg = am.Config(28, 2, 100.0)
    t = cfg.total
    sims = []
    for _ in range(2):
        sim = am.Sim(cfg, am.SIM_WAVE, slots=64, mode=am.MODE_BATCHED)
        for c in range(8):
            sim.add_node(0, c)
        first = int(sim.state()["children"][0])
        for c in range(8):
            sim.add_node(first, c)
        gone = [int(v) for v in sim.state()["children"][first * 8: first * 8 + 4]]
        sim.remove_nodes(gone)
        sim.synchronize()
        st = sim.state()
        used = st["used_slots"]
        assert used == 17 and np.count_nonzero(st["positions"][:used] == 0xFFFFFFFF) == 4
        rng = np.random.default_rng(3)
        for which, far in ((am.Sim.OLD, 1e6), (am.Sim.NEW, 0.)):   # the live domains nearly flat: the tree stays
            f = (.5 + 1e-4 * rng.random((used, t ** 3))).astype(np.float32)
            f[gone] += np.float32(far)
            sim.tensor(which)[: used * t ** 3].copy_(torch.from_numpy(f.reshape(-1)))
        torch.cuda.synchronize()
        sims.append(sim)
    whole, phased = sims
    whole.timestep()
    while True:
        for ph in PHASES:
            phased.phase(getattr(am, "PHASE_" + ph))
        if phased.state()["timer"] == 0:
            break
    whole.synchronize()
    phased.synchronize()
    a, b = whole.state(), phased.state()
    assert all(np.array_equal(a[k], b[k]) for k in a) and a["used_slots"] == used
    for which in (am.Sim.NEW, am.Sim.OLD):
        x, y = (s.tensor(which)[: used * t ** 3].cpu().numpy().view(np.uint32) for s in sims)
        assert np.count_nonzero(x != y) == 0, f"buffer {which}: {np.count_nonzero(x != y)} words differ"
    whole.close()
    phased.close()
