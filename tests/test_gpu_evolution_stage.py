"""The fused RK stage of the BSSN evolution (kernels_evolve_stage.cu) at both of its tile forms: 16^3
domains few enough for the small tiles (9 domains) and enough for the large ones (73), with the
Gamma-driver on (every field visited, the driver's too) and off."""
from __future__ import annotations

import pytest

import cases
from test_evolution_cpu import OracleEvolution, evo_params
from test_gpu_evolution import compare, gpu_sim, gpu_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,shift", [(1, 1), (2, 1), (2, 0)])
def test_stage_tiles_match_fp64(am, cuda, orc, depth, shift):
    """Periodic gauge wave (A = 0.05), one root step of the graph replay against the FP64 oracle: every
    field within 1e-4 of its scale, the tolerance of the same comparison on 8^3 and 32^3 domains
    (single-precision rounding of the state, about 2^-24 / (dx^2 / dt))."""
    ev = am.Evolution(slicing=am.SLICING_1PLUSLOG, shift=shift, eta=2.0, ko_sigma=0.1, cfl=0.25, periodic=1)
    data = am.InitialData(kind=am.ID_GAUGE_WAVE, amplitude=0.05, wavelength=1.0)
    sim = gpu_sim(am, 16, 1.0, lambda o: cases.tree_uniform(o, depth), am.SIM_BSSN_EVOLVE, ev, data, am.MODE_GRAPH,
                  slots=sum(8 ** d for d in range(depth + 1)))
    sim.timestep()
    sim.synchronize()
    st = sim.state()
    gpu = gpu_state(am, sim, 24)
    sim.close()
    ref = OracleEvolution(orc, evo_params(orc, 16, 1.0, slicing=0, shift=shift, id_kind=1, amplitude=0.05, wavelength=1.0), st)
    ref.timestep(1)
    compare(gpu, ref.new, st, 16, 1e-4, f"gauge wave, depth {depth}, shift {shift}")
