"""The smallest meshes in z: on three planes the zero-flux stencil of a z wall
(bc.f90:345-390) reaches the other wall's face, which the BC list updates
bottom first.  Both schedules and every form of a pass against the oracle,
bit for bit."""
import numpy as np
import pytest

import nimgpu
from nimgpu import _abi, config
import oracle as O

pytestmark = pytest.mark.gpu

STATE = [
    _abi.FACES_U, _abi.FACES_V, _abi.FACES_W, _abi.FACES_P, _abi.FACES_T,
    _abi.MESHES_U, _abi.MESHES_V, _abi.MESHES_W, _abi.MESHES_T,
]
DIMS = [(6, 3, 3), (12, 6, 3), (33, 5, 3), (40, 24, 3)]


def pair(dims, oracle_order, **over):
    case = config.small_case(*dims)
    params = case.params(**over)
    mesh = nimgpu.Mesh(case.mesh_params())
    gpu = nimgpu.NimSolver(mesh, params)
    gpu.initialize_nse()
    ref = O.Oracle(mesh, params, schedule=oracle_order)
    ref.init()
    gpu.add_temperature_noise(case.noise, case.seed)
    nimgpu.apply_temperature_noise(ref.get, ref.set, mesh, case.noise, case.seed)
    return gpu, ref


def same_fields(gpu, ref):
    for f in STATE:
        a = gpu.download(f)
        assert np.array_equal(a, ref.get(f, a.size)), f


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("schedule,formulation", [(0, 2), (1, 2), (1, 1)])
def test_passes_match_the_oracle(dims, schedule, formulation):
    gpu, ref = pair(dims, O.PARALLEL if schedule == 0 else O.SEQUENTIAL,
                    schedule=_abi.SCHEDULE_PARALLEL if schedule == 0 else _abi.SCHEDULE_REFERENCE,
                    formulation=formulation)
    gpu.calculate_velocity_nim_constants()
    ref.begin_step()
    for n in (1, 3):
        g, r = gpu.iterate(n), ref.iterate(n)
        assert (g.err_u, g.err_v, g.err_w, g.err_p, g.err_T) == (r.err_u, r.err_v, r.err_w, r.err_p, r.err_T)
        same_fields(gpu, ref)
    gpu.close()


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("loop", ["on", "off"])
def test_steps_match_the_oracle(monkeypatch, dims, loop):
    monkeypatch.setenv("NIM_PASS_LOOP", loop)
    gpu, ref = pair(dims, O.PARALLEL)
    got = gpu.solve_nse(2)
    _, want = ref.step(2)
    assert [g.iters for g in got] == [r.iters for r in want]
    same_fields(gpu, ref)
    gpu.close()


def test_mixed_precision_forms_agree(monkeypatch):
    out = []
    for loop in ("on", "off"):
        monkeypatch.setenv("NIM_PASS_LOOP", loop)
        gpu, _ = pair((40, 24, 3), O.PARALLEL, precision=_abi.PRECISION_MIXED)
        recs = gpu.solve_nse(2)
        out.append(([(r.iters, r.iters_fp32) for r in recs], [gpu.download(f) for f in STATE]))
        gpu.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
