"""Contexts advanced by several host threads at once: the inner loop runs as
one cooperative launch while the loops of all advancing calls fit the device
side by side, and as launches, which overlap, where they do not.  The same
bits whichever it is, in the middle of a step too."""
import threading

import numpy as np
import pytest

import nimgpu
from nimgpu import _abi, config

pytestmark = pytest.mark.gpu

STATE = [
    _abi.FACES_U, _abi.FACES_V, _abi.FACES_W, _abi.FACES_P, _abi.FACES_T,
    _abi.MESHES_U, _abi.MESHES_V, _abi.MESHES_W, _abi.MESHES_T, _abi.MESHES_P,
]


def solver(dims, seed, **over):
    case = config.small_case(*dims, **({"seed": seed}))
    s = nimgpu.NimSolver(nimgpu.Mesh(case.mesh_params()), case.params(**over))
    s.initialize_nse()
    s.add_temperature_noise(case.noise, case.seed)
    return s


def advance(s, n):
    before = s.launch_count()
    recs = s.solve_nse(n)
    return [(r.iters, r.iters_fp32, r.nu_inner, r.nu_outer, r.err_p) for r in recs], s.launch_count() - before


def side_by_side(solvers, n):
    out = [None] * len(solvers)
    gate = threading.Barrier(len(solvers))

    def work(i):
        gate.wait()
        out[i] = advance(solvers[i], n)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(solvers))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return out


@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_loops_that_fill_the_device_give_way_to_launches(monkeypatch, precision):
    for name in ("NIM_PASS_LOOP", "NIM_CELL_SWEEP", "NIM_FACE_SWEEP"):
        monkeypatch.delenv(name, raising=False)
    dims, n = (48, 48, 32), 4
    alone = [solver(dims, 7 + i, precision=precision) for i in range(4)]
    together = [solver(dims, 7 + i, precision=precision) for i in range(4)]
    want = [advance(s, n) for s in alone]
    got = side_by_side(together, n)
    assert [g[0] for g in got] == [w[0] for w in want]
    # a pass is eight launches, a loop one for all its passes
    assert sum(g[1] for g in got) > 4 * sum(w[1] for w in want)
    for s, t in zip(alone, together):
        for f in STATE:
            assert np.array_equal(s.download(f), t.download(f)), f
    # alone again: loops again
    last = advance(together[0], 1)
    assert last == advance(alone[0], 1)
    for s in alone + together:
        s.close()


def test_loops_that_fit_side_by_side_stay_loops(monkeypatch):
    for name in ("NIM_PASS_LOOP", "NIM_CELL_SWEEP", "NIM_FACE_SWEEP"):
        monkeypatch.delenv(name, raising=False)
    alone = [solver((36, 6, 12), 3 + i) for i in range(3)]
    together = [solver((36, 6, 12), 3 + i) for i in range(3)]
    assert side_by_side(together, 3) == [advance(s, 3) for s in alone]
    for s in alone + together:
        s.close()
