"""The bounded grid barrier of the inner loop's cooperative form:
nim_gpu_selftest_barrier_timeout waits for an arrival that does not come (no
block waits for another to be resident) and reports the status the device
recorded; afterwards the context must still step normally, in a loop."""
import pytest

import nimgpu
from nimgpu import _abi, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tries", [1, 1000])
def test_bounded_barrier_reports_timeout_and_the_context_stays_usable(monkeypatch, tries):
    monkeypatch.setenv("NIM_PASS_LOOP", "on")
    case = config.small_case(16, 6, 6)
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params())
    s.initialize_nse()
    s.add_temperature_noise(case.noise, case.seed)
    assert s.lib.nim_gpu_selftest_barrier_timeout(s._h, tries) == _abi.NIM_ERR_TIMEOUT
    assert s.lib.nim_gpu_selftest_barrier_timeout(s._h, 0) == _abi.NIM_ERR_BAD_ARG
    recs = s.solve_nse(2)
    assert all(r.status == _abi.NIM_OK and r.iters > 1 for r in recs)
    s.close()
