"""A kernel launch that the runtime refuses: the call that made it says so (the estimator's passes, the simulations'
timesteps and the constraint norms; each launch of a call refused in turn)."""
from __future__ import annotations

import pytest

import fake_cuda

SCAN = """
L = am.load()
N = 70
feat, tgt = np.zeros((N, 3, 512), np.float32), np.zeros(N, np.float32)
grads, pred, loss, norms = np.zeros(L.amr_estimator_param_count(), np.float32), np.zeros(N, np.float32), ctypes.c_float(), (ctypes.c_double * 5)()
from adaptivemesh_gb300.estimator import Estimator
estimator = lambda: Estimator(128)
def sim(kind, *cfg):
    def make():
        s = am.Sim(am.Config(*cfg), kind, slots=16, mode=am.MODE_BATCHED)
        cases.tree_wave(s)
        return s
    return make
calls = {
    "forward": (estimator, lambda e: L.amr_estimator_forward(e.h, feat.ctypes.data, N, pred.ctypes.data)),
    "gradients": (estimator, lambda e: L.amr_estimator_gradients(e.h, feat.ctypes.data, tgt.ctypes.data, N, grads.ctypes.data, ctypes.byref(loss))),
    "train_step": (estimator, lambda e: L.amr_estimator_train_step(e.h, feat.ctypes.data, tgt.ctypes.data, N, 1e-3, ctypes.byref(loss))),
    "set_params": (estimator, lambda e: L.amr_estimator_set_params(e.h, grads.ctypes.data)),
    "bssn": (sim(am.SIM_BSSN, 16, 3, 1.0), lambda s: L.amr_sim_timestep(s.h)),
    "simplewave": (sim(am.SIM_WAVE, 28, 2, 1.0), lambda s: L.amr_sim_timestep(s.h)),
    "wave_rk4": (sim(am.SIM_WAVE_RK4, 8, 3, 1.0), lambda s: L.amr_sim_timestep(s.h)),
    "evolve": (sim(am.SIM_BSSN_EVOLVE, 8, 3, 1.0), lambda s: L.amr_sim_timestep(s.h)),
    "norms": (sim(am.SIM_BSSN_EVOLVE, 8, 3, 1.0), lambda s: L.amr_sim_constraint_norms(s.h, ctypes.c_float(0), norms)),
}
out = {}
for name, (make, call) in calls.items():
    h = make()
    assert call(h) == 0
    fake.fake_reset(0)
    assert call(h) == 0
    n = fake.fake_launches()
    bad = []
    for k in range(1, n + 1):
        h = make()
        call(h)
        fake.fake_reset(k)
        status, kernel = call(h), fake.fake_kernel(k - 1).decode()
        fake.fake_reset(0)
        if SECOND:
            status = call(make()) == 0   # the next call, of another object, is not blamed
        else:
            fake.cudaGetLastError()
        if not status:
            bad.append(kernel)
    out[name] = (n, bad)
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def scan(am, tmp_path_factory):
    return lambda second: fake_cuda.run(tmp_path_factory.mktemp("fake"), f"SECOND = {second}\n" + SCAN)


def test_every_refused_launch_is_reported(scan):
    out = scan(False)
    assert all(n > 0 for n, _ in out.values())
    assert not any(bad for _, bad in out.values()), out


def test_a_refused_launch_is_reported_once(scan):
    out = scan(True)
    assert not any(bad for _, bad in out.values()), out
