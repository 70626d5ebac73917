"""The reference order on meshes whose levels are narrow while the mesh is
long in one direction, on both sides of the limit of the skewed copies
(nim_reference_form): two passes of the loop body, bit for bit the oracle's
sequential order (nse.f90:131-160)."""
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


@pytest.mark.parametrize("dims,formulation,form", [
    ((24, 24, 200), 2, 2), ((24, 24, 200), 1, 2), ((6, 10, 150), 2, 2), ((6, 90, 30), 2, 2), ((7, 8, 160), 1, 2),
    ((6, 10, 900), 2, 1), ((7, 9, 850), 1, 1), ((24, 24, 600), 2, 1), ((24, 200, 110), 2, 1)])
def test_two_passes_match_the_sequential_oracle(dims, formulation, form):
    assert _abi.gpu_lib().nim_reference_form(*dims, None) == form
    case = config.small_case(*dims)
    params = case.params(schedule=_abi.SCHEDULE_REFERENCE, formulation=formulation)
    mesh = nimgpu.Mesh(case.mesh_params())
    gpu = nimgpu.NimSolver(mesh, params)
    gpu.initialize_nse()
    ref = O.Oracle(mesh, params, schedule=O.SEQUENTIAL)
    ref.init()
    gpu.add_temperature_noise(case.noise, case.seed)
    nimgpu.apply_temperature_noise(ref.get, ref.set, mesh, case.noise, case.seed)
    gpu.calculate_velocity_nim_constants()
    ref.begin_step()
    g, r = gpu.iterate(2), ref.iterate(2)
    assert (g.err_u, g.err_v, g.err_w, g.err_p, g.err_T) == (r.err_u, r.err_v, r.err_w, r.err_p, r.err_T)
    for f in STATE:
        a = gpu.download(f)
        assert np.array_equal(a, ref.get(f, a.size)), f
    gpu.close()
