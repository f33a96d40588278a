"""Device memory of a BSSN evolution: per field three padded buffers and the accumulator, the four constraints and the
four planes that the tuning call writes; nothing for derivatives, which no kernel stores."""
from __future__ import annotations

import pytest

import fake_cuda


@pytest.mark.parametrize("n,slots", [(8, 200), (16, 73)])
def test_memory_per_cell(am, tmp_path, n, slots):
    out = fake_cuda.run(tmp_path, f"""
        fake.fake_reset(0)
        sim = am.Sim(am.Config({n}, 3, 1.0), am.SIM_BSSN_EVOLVE, slots={slots}, mode=am.MODE_GRAPH)
        out = [fake.fake_allocated()]
        p, c = ctypes.c_void_p(), ctypes.c_uint64()
        for comp in range(5):
            out.append(am.load().amr_sim_buffer(sim.h, sim.DERIVS, comp, ctypes.byref(p), ctypes.byref(c)) == 0)
        print(json.dumps(out))
    """)
    fields = 4 * slots * (24 * (3 * (n + 6) ** 3 + n ** 3) + 8 * n ** 3)
    assert fields <= out[0] <= fields + (1 << 14) * slots, (out[0], fields)
    assert out[1:] == [True] * 4 + [False]
