"""max_iters bounds the passes of a step that ran, both phases of a mixed
step together (nim_params.max_iters, include/nim_gpu.h), in every form the
inner loop takes: a step that cannot converge stops after exactly that many,
whatever was queued beyond a phase's end."""
import pytest

import nimgpu
from nimgpu import _abi, config

pytestmark = pytest.mark.gpu

# the temperature's test cannot hold: FP32 passes end once its changes stop
# falling (rounding), FP64 passes go on to the cap
NEVER = dict(tol_u=1e-3, tol_v=1e-3, tol_w=1e-3, tol_p=1e-2, tol_T=-1.0)


def solver(cap, **over):
    case = config.small_case(16, 8, 8)
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params(max_iters=cap, **over))
    s.initialize_nse()
    s.add_temperature_noise(case.noise, case.seed)
    return s


@pytest.mark.parametrize("loop", ["on", "off"])
@pytest.mark.parametrize("cap", [37, 600, 1100])
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_a_step_runs_to_its_cap(monkeypatch, loop, cap, precision):
    """The second step launches ahead by the first one's counts."""
    monkeypatch.setenv("NIM_PASS_LOOP", loop)
    s = solver(cap, precision=precision, **NEVER)
    for _ in range(2):
        s.calculate_velocity_nim_constants()
        rec = s.integrate_nse(raise_on_error=False)
        assert rec.status == _abi.NIM_ERR_NOT_CONVERGED
        assert rec.iters == cap
        if precision == _abi.PRECISION_MIXED and cap >= 600:
            # the FP64 phase takes more than one launch of a loop
            assert 0 < rec.iters_fp32 < cap - 256
        s.update_time_step()
    s.close()


@pytest.mark.parametrize("fused", [False, True])
def test_batches_run_to_their_caps(fused):
    caps = [150, 700, 700, 41]
    ctx = [solver(c, precision=_abi.PRECISION_MIXED, **NEVER) for c in caps]
    recs = nimgpu.batch_step(ctx, 1, fused=fused, raise_on_error=False)
    assert [r[0].iters for r in recs] == caps
    assert all(r[0].status == _abi.NIM_ERR_NOT_CONVERGED for r in recs)
    for s in ctx:
        s.close()
