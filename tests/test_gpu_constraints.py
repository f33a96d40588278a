"""The constraint pass (kernels_evolve_constraints.cu) at each compiled size, on a tree with covered,
partly covered and leaf domains: the tile depth does not change a bit of the fields, and the norms are
the double-precision reduction of those fields."""
from __future__ import annotations

import numpy as np
import pytest

import cases
from test_gpu_evolution import gpu_sim

pytestmark = pytest.mark.gpu


def tree_partial(o):
    """Uniform depth 1, then one of its domains refined in all octants and one in two of them."""
    cases.tree_uniform(o, 1)
    ch = o.state()["children"]
    for octant in range(8):
        o.add_node(int(ch[0]), octant)
    for octant in (0, 5):
        o.add_node(int(ch[6]), octant)


@pytest.mark.parametrize("n", [8, 16, 32])
def test_constraint_tiles_and_norms(am, cuda, n):
    """A gauge wave.  Every cell's arithmetic is the same at any tile depth, so the planes
    that the tuning call leaves (its last depth) equal the default's bit for bit.  The norms sum n^3 terms a
    domain in double: 1e-12 of the same sum in another order (2^-53 a term, 6e5 terms at most)."""
    ev = am.Evolution(slicing=am.SLICING_1PLUSLOG, shift=0, ko_sigma=0.1, cfl=0.25, periodic=1)
    data = am.InitialData(kind=am.ID_GAUGE_WAVE, amplitude=0.05, wavelength=1.0)
    sim = gpu_sim(am, n, 1.0, tree_partial, am.SIM_BSSN_EVOLVE, ev, data,
                  am.MODE_GRAPH, slots=20)
    sim.timestep()
    import torch
    norms = sim.constraint_norms()
    st = sim.state()
    used = st["used_slots"]
    get = lambda which, c: sim.tensor(which, c, dtype=torch.float32)[: used * n ** 3].cpu().numpy().reshape(used, n, n, n)  # noqa: E731
    cons = [get(am.Sim.CONSTRAINTS, c) for c in range(4)]
    sim.autotune(1)
    sim.synchronize()
    planes = [get(am.Sim.DERIVS, c) for c in range(4)]
    tuned = sim.constraint_norms()
    children = np.asarray(st["children"]).reshape(-1, 8)[:used]
    live = np.asarray(st["positions"])[:used] != 0xFFFFFFFF
    mask = np.zeros((used, n, n, n), bool)
    h = n // 2
    for s in range(used):
        if not live[s]:
            continue
        for o in range(8):
            if children[s, o] == -1:
                x, y, z = (o & 1) * h, (o >> 1 & 1) * h, (o >> 2) * h
                mask[s, z:z + h, y:y + h, x:x + h] = True
    evolved = [s for s in range(used) if mask[s].any()]
    for c in range(4):
        assert np.array_equal(planes[c][evolved], cons[c][evolved]), f"component {c} differs between tile depths"
    hh = cons[0][mask].astype(np.float64)
    m2 = sum(cons[c][mask].astype(np.float64) ** 2 for c in (1, 2, 3))
    want = {"H_l2": np.sqrt((hh * hh).mean()), "H_max": np.abs(hh).max(), "M_l2": np.sqrt(m2.mean()), "M_max": np.sqrt(m2.max())}
    for got in (norms, tuned):
        assert got["cells"] == mask.sum()
        for k, w in want.items():
            assert abs(got[k] - w) <= 1e-12 * w, (k, got[k], w)
    sim.close()
