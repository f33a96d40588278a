"""The evolutions' restriction (k_evo_restrict) at each compiled size and both field counts, on a tree with
covered, partly covered and leaf domains, against the 4-point midpoint rule in double precision."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_constraints import tree_partial
from test_gpu_evolution import gpu_sim

pytestmark = pytest.mark.gpu


def midpoint(a, axis):
    """(-1, 9, 9, -1) / 16 along an axis, every second position."""
    m = a.shape[axis]
    t = [np.take(a, np.arange(k, m - 3 + k, 2), axis) for k in range(4)]
    return (9 * (t[1] + t[2]) - t[0] - t[3]) / 16


@pytest.mark.parametrize("kind", ["bssn", "wave"])
@pytest.mark.parametrize("n", [8, 16, 32])
def test_restriction_matches_midpoint_rule(am, cuda, n, kind):
    """Random fields of magnitude up to 1: covered cells to 1.2e-6 (four roundings an axis, of at most 2^-24 as
    every value stays below 2, grown by later axes to at most 1.25^2: 12 * 2^-24 * 1.57 = 1.13e-6), all
    other cells, ghosts included, exactly."""
    import torch
    bssn = kind == "bssn"
    ev = am.Evolution(slicing=am.SLICING_1PLUSLOG, shift=0, ko_sigma=0.1, cfl=0.25, periodic=1)
    data = am.InitialData(kind=am.ID_GAUGE_WAVE if bssn else am.ID_GAUSSIAN_PULSE, amplitude=0.05, wavelength=1.0, width=0.1)
    sim = gpu_sim(am, n, 1.0, tree_partial, am.SIM_BSSN_EVOLVE if bssn else am.SIM_WAVE_RK4, ev, data, am.MODE_BATCHED, slots=20)
    st = sim.state()
    used, t, h = st["used_slots"], n + 6, n // 2
    g = torch.Generator(device="cuda").manual_seed(n)
    new = []
    for f in range(24 if bssn else 2):
        x = sim.tensor(am.Sim.NEW_STATE, f)
        x.copy_(torch.rand(x.numel(), generator=g, device="cuda") * 2 - 1)
        new.append(x[: used * t ** 3].cpu().numpy().reshape(used, t, t, t))
    torch.cuda.synchronize()
    sim.phase(am.PHASE_COPY_BACK)
    sim.synchronize()
    children = np.asarray(st["children"]).reshape(-1, 8)
    for f, v in enumerate(new):
        old = sim.tensor(am.Sim.OLD_STATE, f)[: used * t ** 3].cpu().numpy().reshape(used, t, t, t)
        for s in range(used):
            covered = np.zeros((t, t, t), bool)
            for o in range(8):
                if children[s, o] == -1:
                    continue
                at = tuple(slice(3 + (o >> a & 1) * h, 3 + (o >> a & 1) * h + h) for a in (2, 1, 0))
                c = v[children[s, o]][2:n + 4, 2:n + 4, 2:n + 4].astype(np.float64)
                want = midpoint(midpoint(midpoint(c, 2), 1), 0)
                covered[at] = True
                assert np.abs(old[s][at] - want).max() <= 1.2e-6, (f, s, o)
            assert np.array_equal(old[s][~covered], v[s][~covered]), (f, s)
    sim.close()
