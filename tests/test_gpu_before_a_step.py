"""Passes of the loop body before the first nim_gpu_begin_step: the velocity
constants are still zero, every update divides by them, and the call reports
it, whatever the schedule and formulation."""
import ctypes as C

import pytest

import nimgpu
from nimgpu import _abi, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(12, 6, 6), (36, 14, 14), (90, 70, 60)])
@pytest.mark.parametrize("schedule", [_abi.SCHEDULE_PARALLEL, _abi.SCHEDULE_REFERENCE])
@pytest.mark.parametrize("formulation", [1, 2])
def test_passes_without_a_steps_constants_are_not_finite(dims, schedule, formulation):
    case = config.small_case(*dims)
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params(schedule=schedule, formulation=formulation))
    s.initialize_nse()
    s.add_temperature_noise(case.noise, case.seed)
    rec = _abi.StepStats()
    assert s.lib.nim_gpu_iterate(s._h, 2, C.byref(rec)) == _abi.NIM_ERR_NONFINITE
    # a step of its own is fine from the initial state
    s.initialize_nse()
    s.calculate_velocity_nim_constants()
    assert s.lib.nim_gpu_iterate(s._h, 2, C.byref(rec)) == _abi.NIM_OK
    s.close()
