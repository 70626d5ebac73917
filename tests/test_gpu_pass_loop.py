"""The forms a parallel pass takes by mesh size and shape (include/nim_gpu.h,
nim_gpu_create): the inner loop as one cooperative launch against launches of
a graph, and the sweeps' blocks over patches of the plane against runs of it
in cell order.  Every form gives the same bits: iteration counts, Nusselt
numbers and every field over whole steps, the oracle's among them."""
import threading

import numpy as np
import pytest

import nimgpu
from nimgpu import _abi, config
import oracle as O

pytestmark = pytest.mark.gpu

STATE = [
    _abi.FACES_U, _abi.FACES_V, _abi.FACES_W, _abi.FACES_P, _abi.FACES_T,
    _abi.MESHES_U, _abi.MESHES_V, _abi.MESHES_W, _abi.MESHES_T, _abi.MESHES_P,
]


def steps(case, n=2, **over):
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params(**over))
    s.initialize_nse()
    s.add_temperature_noise(case.noise, case.seed)
    recs = s.solve_nse(n)
    out = [(r.iters, r.iters_fp32, r.nu_inner, r.nu_outer, r.err_u, r.err_p, r.err_T) for r in recs]
    fields = [s.download(f) for f in STATE]
    launched = s.launch_count()
    s.close()
    return out, fields, launched


def equal(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)


# the smallest mesh, one cell past a warp, a block's edge, odd and ragged,
# several turns of a block (pairs and one cell a thread), whole warps
@pytest.mark.parametrize("dims", [(6, 3, 4), (33, 4, 5), (32, 4, 4), (45, 37, 29), (64, 48, 40), (63, 50, 41), (96, 8, 6)])
@pytest.mark.parametrize("over", [dict(), dict(precision=_abi.PRECISION_MIXED), dict(dpdx_tolerance=1, tol_p=1e-4)],
                         ids=["fp64", "mixed", "dpdx"])
def test_loop_and_launches_are_bitwise_equal(monkeypatch, dims, over):
    case = config.small_case(*dims)
    monkeypatch.setenv("NIM_PASS_LOOP", "off")
    plain = steps(case, **over)
    monkeypatch.setenv("NIM_PASS_LOOP", "on")
    loop = steps(case, **over)
    equal(plain, loop)
    assert loop[2] < plain[2]  # whole loops in a few launches


def test_loop_matches_the_oracle_and_respects_the_cap(monkeypatch):
    monkeypatch.delenv("NIM_PASS_LOOP", raising=False)
    case = config.small_case(19, 7, 8)
    mesh, params = nimgpu.Mesh(case.mesh_params()), case.params()
    ref = O.Oracle(mesh, params, schedule=O.PARALLEL)
    ref.init()
    nimgpu.apply_temperature_noise(ref.get, ref.set, mesh, case.noise, case.seed)
    _, r = ref.step(2)
    got, fields, _ = steps(case)
    assert [g[0] for g in got] == [x.iters for x in r]
    for f, v in zip(STATE, fields):
        assert np.array_equal(v, ref.get(f, v.size)), f
    for cap in (1, 5):
        s = nimgpu.NimSolver(mesh, case.params(max_iters=cap))
        s.initialize_nse()
        s.calculate_velocity_nim_constants()
        rec = s.integrate_nse(raise_on_error=False)
        assert rec.status == _abi.NIM_ERR_NOT_CONVERGED and rec.iters == cap
        s.close()


def test_loop_reports_a_nonfinite_pass(monkeypatch):
    monkeypatch.setenv("NIM_PASS_LOOP", "on")
    case = config.small_case(12, 6, 6)
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params())
    s.initialize_nse()
    t = s.download(_abi.FACES_T)
    t[s.mesh.interior_faces.nonzero()[0][5]] = np.nan
    s.upload(_abi.FACES_T, t)
    s.calculate_velocity_nim_constants()
    assert s.integrate_nse(raise_on_error=False).status == _abi.NIM_ERR_NONFINITE
    s.close()


def test_loops_of_several_threads_side_by_side(monkeypatch):
    """Contexts of four host threads, each with its own stream and loop."""
    monkeypatch.delenv("NIM_PASS_LOOP", raising=False)
    cases = [config.small_case(*d) for d in ((36, 6, 12), (45, 30, 20), (24, 12, 12), (48, 24, 20))]
    want = [steps(c, 3) for c in cases]
    got = [None] * len(cases)

    def work(i):
        got[i] = steps(cases[i], 3)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(want, got):
        equal(a, b)


# sweeps whose patches would idle more than a tenth of the threads run in
# cell order: n_theta past a warp, pairs and groups of four past it, rows
@pytest.mark.parametrize("dims", [(40, 9, 6), (66, 9, 5), (132, 6, 6), (100, 12, 5), (35, 9, 7)])
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
def test_cell_order_sweeps_match_the_oracle(monkeypatch, dims, precision):
    monkeypatch.setenv("NIM_PASS_LOOP", "off")
    case = config.small_case(*dims)
    got, fields, _ = steps(case, precision=precision)
    if precision == _abi.PRECISION_FP64:
        mesh, params = nimgpu.Mesh(case.mesh_params()), case.params()
        ref = O.Oracle(mesh, params, schedule=O.PARALLEL)
        ref.init()
        nimgpu.apply_temperature_noise(ref.get, ref.set, mesh, case.noise, case.seed)
        _, r = ref.step(2)
        assert [g[0] for g in got] == [x.iters for x in r]
        for f, v in zip(STATE, fields):
            assert np.array_equal(v, ref.get(f, v.size)), f
    else:  # the loop's one-cell float sweeps
        monkeypatch.setenv("NIM_PASS_LOOP", "on")
        equal((got, fields), steps(case, precision=precision))
