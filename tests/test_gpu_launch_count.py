"""nim_gpu_launch_count against the kernels a pass of the reference order
launches: one per entry of nim_gpu_profile_iterations, the walls' fixed terms
beside their sweep, and the six copies around the skewed sweeps."""
import pytest

import nimgpu
from nimgpu import _abi, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,form", [((12, 6, 6), 0), ((90, 70, 60), 1), ((36, 14, 14), 2)])
@pytest.mark.parametrize("over", [dict(), dict(dpdx_tolerance=1, tol_p=1e-4)], ids=["plain", "dpdx"])
def test_launches_of_a_reference_order_pass(dims, form, over):
    assert _abi.gpu_lib().nim_reference_form(*dims, None) == form
    case = config.small_case(*dims)
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params(schedule=_abi.SCHEDULE_REFERENCE, **over))
    s.initialize_nse()
    s.calculate_velocity_nim_constants()
    names = s.profile_iterations(1)
    before = s.launch_count()
    s.iterate(3)
    assert s.launch_count() - before == 3 * (len(names) + 1 + (6 if form == 2 else 0))
    s.close()
