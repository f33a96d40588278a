"""The ghost layers that an RK stage of the BSSN evolution writes for its neighbours (EvoArgs::feed), with states that
vary along all three axes: every tile form and number of fed axes, on periodic and on refined trees."""
from __future__ import annotations

import numpy as np
import pytest

import cases
from test_evolution_cpu import OracleEvolution, evo_params
from test_gpu_evolution import compare, gpu_sim, gpu_state

pytestmark = pytest.mark.gpu

TREES = {"uniform1": (lambda o: cases.tree_uniform(o, 1), 9), "uniform2": (lambda o: cases.tree_uniform(o, 2), 73),
         "uniform3": (lambda o: cases.tree_uniform(o, 3), 585), "uneven": (cases.tree_uneven, 64),
         "random4": (lambda o: cases.tree_random(o, 4, 0.3, 0), 200)}
PHASES = ("COPY_BACK", "MODIFY_NODES", "PREDICTOR", "COPY_BOUNDS", "CORRECTOR", "INCREMENT_TIMER")


def varied_sim(am, n, tree, periodic, seed):
    """All three state buffers hold the same sums of periodic modes of the unit box, amplitude about 1e-2 in every
    field, ghost layers included; none is constant along an axis."""
    import torch
    build, slots = TREES[tree]
    ev = am.Evolution(slicing=am.SLICING_1PLUSLOG, shift=1, eta=2.0, ko_sigma=0.1, cfl=0.25, periodic=periodic)
    sim = gpu_sim(am, n, 1.0, build, am.SIM_BSSN_EVOLVE, ev, am.InitialData(kind=am.ID_FLAT), am.MODE_BATCHED, slots=slots)
    st = sim.state()
    xyz = 2 * np.pi * cases.cell_coordinates(st["positions"], st["used_slots"], n, 3, 1.0).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    fields = []
    for f in range(24):
        k = rng.integers(1, 3, (2, 3)) * rng.choice((-1, 1), (2, 3))
        ph = rng.uniform(0, 2 * np.pi, 2)
        fields.append((5e-3 * (np.cos(xyz @ k[0] + ph[0]) + np.cos(xyz @ k[1] + ph[1]))).astype(np.float32))
        for which in (sim.OLD_STATE, sim.NEW_STATE, sim.STAGE):
            sim.tensor(which, f, torch.float32)[: len(xyz)].copy_(torch.from_numpy(fields[-1]))
    torch.cuda.synchronize()
    return sim, st, fields


@pytest.mark.parametrize("n,tree,periodic", [(8, "uniform1", 1), (8, "uniform3", 1), (8, "random4", 0), (16, "uniform1", 1),
                                             (16, "uniform1", 0), (16, "uniform2", 1), (16, "uneven", 0), (16, "random4", 0),
                                             (32, "uniform1", 1), (32, "uniform2", 1), (32, "uneven", 0)])
def test_fed_ghosts_equal_the_filled(am, cuda, n, tree, periodic):
    """Two root steps by timestep(), whose last stage feeds its neighbours, and by the phases called one by one, where
    the fill copies every ghost layer: each padded cell of the state, edges and corners included, bit for bit."""
    import torch
    whole, st, _ = varied_sim(am, n, tree, periodic, 10 * n + periodic)
    phased, _, _ = varied_sim(am, n, tree, periodic, 10 * n + periodic)
    for _ in range(2):
        whole.timestep()
        while True:
            for ph in PHASES:
                phased.phase(getattr(am, "PHASE_" + ph))
            if phased.state()["timer"] == 0:
                break
    whole.synchronize()
    phased.synchronize()
    cells = st["used_slots"] * (n + 6) ** 3
    for f in range(24):
        a, b = (s.tensor(s.NEW_STATE, f)[:cells].view(torch.int32) for s in (whole, phased))
        differ = int((a != b).sum())
        assert differ == 0, f"field {f}: {differ} of {cells} cells differ"
    if periodic and tree == "uniform1":   # all faces are fed: the fill's launches fall away in timestep()
        assert whole.kernel_launches < phased.kernel_launches
    whole.close()
    phased.close()


@pytest.mark.parametrize("n", [8, 16, 32])
def test_three_axis_feed_matches_fp64(am, cuda, orc, n):
    """A periodic root and 8 children (three fed axes at every size), one root step against the FP64 oracle: every
    padded cell of every field within 1e-4 of its scale, the tolerance of the gauge wave on these sizes.  A layer
    stored at a wrong place of a neighbour is off by the field's own variation, 1e-2, over dx."""
    sim, st, fields = varied_sim(am, n, "uniform1", 1, n)
    sim.timestep()
    sim.synchronize()
    gpu = gpu_state(am, sim, 24)
    sim.close()
    ref = OracleEvolution(orc, evo_params(orc, n, 1.0, slicing=0, shift=1), st)
    for f in range(24):
        for buf in (ref.old, ref.new, ref.stage):
            buf[f][:] = fields[f].astype(np.float64) + am.BSSN_OFFSETS[f]
    ref.timestep(1)
    compare(gpu, ref.new, st, n, 1e-4, f"varied state, {n}^3")
