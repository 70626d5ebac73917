"""The level-by-level sweeps of the reference-order schedule over every form
they take: fields in a block's shared memory or in skewed copies, a level
within a warp, within 256 threads, within 512, in several turns of a block,
and on a cooperative grid; both formulations; theta counts
even and odd, the smallest mesh.  Two passes of the loop body, bit for bit
the oracle's sequential order (nse.f90:131-160)."""
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


def widest_level(nt, nr, nz):
    i, j, k = np.meshgrid(np.arange(nt), np.arange(nr), np.arange(nz), indexing="ij")
    return int(np.bincount((i + 2 * j + 3 * k).ravel()).max())


@pytest.mark.parametrize("dims,lo,hi,formulation", [
    ((6, 3, 4), 1, 32, 2), ((6, 3, 4), 1, 32, 1), ((7, 3, 5), 1, 32, 2),
    ((24, 24, 16), 33, 256, 1), ((41, 29, 24), 257, 512, 2), ((41, 29, 24), 257, 512, 1),
    # the largest that fits a block's shared memory and the smallest that does
    # not, an odd number of faces, narrow levels of a mesh that does not fit
    ((36, 14, 13), 33, 256, 2), ((36, 14, 14), 33, 256, 2), ((21, 9, 7), 1, 64, 2), ((21, 9, 7), 1, 64, 1),
    ((301, 5, 6), 1, 32, 2), ((301, 5, 6), 1, 32, 1),
    ((60, 40, 30), 513, 1024, 2), ((90, 70, 60), 1025, 4000, 2), ((90, 70, 60), 1025, 4000, 1),
])
def test_two_passes_match_the_sequential_oracle(dims, lo, hi, formulation):
    assert lo <= widest_level(*dims) <= hi
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


def test_temperature_branches_of_several_contexts_at_once():
    """Contexts of every form stepping together, each with its pressure and
    temperature sweeps side by side, against the same contexts one at a time."""
    dims = [(36, 14, 13), (41, 29, 24), (90, 70, 60), (21, 9, 7)]

    def make():
        out = []
        for n, m in enumerate(dims):
            case = config.small_case(*m)
            s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()),
                                 case.params(schedule=_abi.SCHEDULE_REFERENCE, formulation=1 + n % 2))
            s.initialize_nse()
            s.add_temperature_noise(case.noise, case.seed + n)
            out.append(s)
        return out

    together, alone = make(), make()
    rec = nimgpu.batch_step(together, 2)
    for s, a, r in zip(together, alone, rec):
        q = a.solve_nse(2)
        assert [x.iters for x in r] == [x.iters for x in q]
        for f in STATE:
            assert np.array_equal(s.download(f), a.download(f)), f
    for s in together + alone:
        s.close()
