"""Workloads of the NIM time advance, for timing it as a user's program runs it.

A run of this framework is a time loop: a host hands the library its restart
arrays, advances time steps (each an inner iteration to the reference's
tolerances) and takes the fields back for its restart file.  run() is that
for one step, through nimgpu's public entry points: upload the
restart state, solve_nse (or batch_step, or the tangent-linear steps), pack
and fetch the restart set (for the tangents: the derivatives).  Every run() of a state starts from the same
restart arrays, so its work does not drift from pass to pass.

The ranges stand for what the framework is used on: enclosures from the
reference's own 36 x 6 x 12 default mesh to a 192 x 192 x 144 cylinder,
theta counts that are even, odd and multiples of four, flows just started
from rest (cell Peclet numbers on the series branch of the NIM coefficients)
and developed convection rolls (the exponential branch), FP64 and mixed
precision, both schedules and formulations, batches of uneven enclosures in
both forms, and forward-mode derivatives.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "nim-conv22-shared_b200"))

import nimgpu  # noqa: E402
from nimgpu import _abi, config  # noqa: E402

# write_restart's arrays in file order (include/nim_gpu.h, NIM_OUTPUT_RESTART):
# five face fields, then nine cell fields
FACE_FIELDS = (_abi.FACES_U, _abi.FACES_V, _abi.FACES_W, _abi.FACES_P, _abi.FACES_T)
CELL_FIELDS = (_abi.MESHES_U, _abi.MESHES_V, _abi.MESHES_W, _abi.MESHES_T,
               _abi.MESHES_U_OLD, _abi.MESHES_V_OLD, _abi.MESHES_W_OLD, _abi.MESHES_T_OLD,
               _abi.MESHES_DILA_OLD)
# the time averages the next step's velocity NIM constants are formed from
AVERAGES = (_abi.MESHES_UT, _abi.MESHES_VT, _abi.MESHES_WT, _abi.MESHES_TT)


def _step(name, shape, Ra, dt, roll, **more):
    nt, nr, nz = shape
    return {"name": name, "kind": "step", "n_theta": nt, "n_r": nr, "n_z": nz, "Ra": Ra, "Pr": 0.71, "dt": dt,
            "roll": roll, "steps": 1, "precision": "fp64", "schedule": "parallel", "formulation": 2, **more}


def listed():
    return [
        # the reference's shipped case as it ships (its mesh, physics and time step), where launches count
        _step("reference-default", (36, 6, 12), 1e5, 1e-2, 0.003, Pr=0.7, geometry="reference", passes=188),
        # the same case in the reference's own Gauss-Seidel order, for runs that have to reproduce its iterates
        _step("reference-order", (36, 6, 12), 1e5, 1e-2, 0.0, Pr=0.7, geometry="reference",
              schedule="reference", passes=56),
        # formulation 1, the reference's other velocity scheme, in the order it needs
        _step("formulation1-order", (24, 24, 16), 1e4, 1e-3, 0.0, schedule="reference", formulation=1, passes=88),
        # the small benchmark cylinder (what a laptop run of the reference solves)
        _step("small-c1", (48, 48, 32), 1e4, 1e-3, 0.003, passes=264),
        # an odd theta count, ragged in every direction
        _step("odd-45x37x29", (45, 37, 29), 1e5, 1e-3, 0.003, passes=291),
        # the benchmark cylinder, just started from rest
        _step("c2-start", (128, 128, 96), 1e5, 5e-4, 0.0, passes=279),
        # a production mesh with n_theta even but no multiple of four, in convection
        _step("ragged-150x101x77", (150, 101, 77), 1e5, 5e-4, 0.001, passes=140),
        # the benchmark cylinder in mixed precision, in convection
        _step("c2-mixed", (128, 128, 96), 1e5, 5e-4, 0.01, precision="mixed", passes=165),
        # the largest: the mixed-precision cylinder of the finest study, at three quarters of its resolution
        _step("large-mixed", (192, 192, 144), 1e6, 2.5e-4, 0.0, precision="mixed", passes=130),
        # a parameter study: uneven enclosures advanced together, FP64, one stream each
        {"name": "batch-streams", "kind": "batch", "n": 16, "a_min": 24, "a_max": 64, "form": "streams",
         "precision": "fp64", "steps": 1, "batch_seed": 2024, "passes": 170},
        # the same study in mixed precision, every pass kernel launched once for all
        {"name": "batch-fused-mixed", "kind": "batch", "n": 16, "a_min": 24, "a_max": 64, "form": "fused",
         "precision": "mixed", "steps": 1, "batch_seed": 2024, "passes": 170},
        # forward-mode derivative d/dRa on the sensitivity mesh
        _step("tangent-c5", (64, 64, 48), 1e5, 1e-3, 0.0, kind="tangent", passes=157),
    ]


def _shape(rng, cells):
    """An anisotropic mesh of about that many cells; theta counts of every remainder."""
    a = (cells / 0.75) ** (1.0 / 3.0)
    nt = max(12, round(a * rng.uniform(0.8, 1.5)))
    nr = max(6, round(a * rng.uniform(0.7, 1.2)))
    return nt, nr, max(6, round(cells / (nt * nr)))


def draw(rng):
    pick = rng.random()
    if pick < 0.60:  # one enclosure, small to large
        shape = _shape(rng, math.exp(rng.uniform(math.log(2.5e3), math.log(2.5e6))))
        return _unnamed(_step("", shape, 10.0 ** rng.uniform(4.0, 5.5), rng.choice((2.5e-4, 5e-4, 1e-3)),
                              rng.choice((0.0, rng.uniform(0.001, 0.01))),
                              precision=rng.choice(("fp64", "fp64", "mixed")), passes=180))
    if pick < 0.72:  # the reference's order
        shape = _shape(rng, math.exp(rng.uniform(math.log(2.5e3), math.log(2e4))))
        return _unnamed(_step("", shape, 10.0 ** rng.uniform(4.0, 5.0), 1e-3, 0.0,
                              schedule="reference", formulation=rng.choice((1, 2, 2)), passes=100))
    if pick < 0.90:  # a parameter study
        lo = rng.randint(16, 32)
        return {"kind": "batch", "n": rng.randint(4, 24), "a_min": lo, "a_max": lo + rng.randint(4, 32),
                "form": rng.choice(("streams", "fused")), "precision": rng.choice(("fp64", "mixed")), "steps": 1,
                "batch_seed": rng.randint(1, 10 ** 6), "passes": 150}
    shape = _shape(rng, math.exp(rng.uniform(math.log(1e4), math.log(3e5))))
    return _unnamed(_step("", shape, 10.0 ** rng.uniform(4.0, 5.0), 1e-3, rng.choice((0.0, 0.003)),
                          kind="tangent", passes=150))


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


def _case_of(case):
    """The framework's run configuration of a single-enclosure case."""
    c = config.Case("case", case["n_theta"], case["n_r"], case["n_z"], Ra=case["Ra"], Pr=case["Pr"], dt=case["dt"],
                    steps=case["steps"])
    over = {"schedule": _abi.SCHEDULE_REFERENCE if case["schedule"] == "reference" else _abi.SCHEDULE_PARALLEL,
            "formulation": case["formulation"],
            "precision": _abi.PRECISION_MIXED if case["precision"] == "mixed" else _abi.PRECISION_FP64}
    if case.get("geometry") == "reference":  # create_hollow's own cylinder, radii and parameters
        mp = config.reference_mesh(n_theta=case["n_theta"], n_r=case["n_r"], n_z=case["n_z"])
        return mp, config.reference_params(Ra=case["Ra"], Pr=case["Pr"], DT=case["dt"], **over)
    return c.mesh_params(), c.params(**over)


def _start(solver, mp, speed, amp, seed):
    """Initial fields: rest with the seeded 1e-6 noise on T, or a convection
    roll of that speed (a divergence-free overturning cell, up along the hot
    hexagon) over the conduction profile, with the same noise."""
    solver.initialize_nse()
    if speed:
        mesh = solver.mesh
        mid = solver.download(_abi.FACES_MID).reshape(mesh.nface, 3)
        cell = mid[mesh.meshes_faces - 1].mean(axis=1)

        def fields(x):
            r = np.hypot(x[:, 0], x[:, 1])
            s = np.clip((r - mp.R_i) / (mp.R_o - mp.R_i), 0.0, 1.0)
            z = x[:, 2] / mp.L
            q = (mp.R_o - mp.R_i) / r
            ur = speed * q * np.sin(math.pi * s) ** 2 * np.sin(2 * math.pi * z)
            w = speed * q * np.sin(2 * math.pi * s) * np.sin(math.pi * z) ** 2
            T = np.clip(np.log(mp.R_o / r) / math.log(mp.R_o / mp.R_i), 0.0, 1.0)
            T = T + 0.2 * (z - 0.5) * np.sin(math.pi * s)
            return ur * x[:, 0] / r, ur * x[:, 1] / r, w, T

        inner = mesh.interior_faces
        for f, v in zip((_abi.FACES_U, _abi.FACES_V, _abi.FACES_W, _abi.FACES_T), fields(mid)):
            solver.upload(f, np.where(inner, v, solver.download(f)))
        for fs, v in zip(((_abi.MESHES_U, _abi.MESHES_U_OLD, _abi.MESHES_UT),
                          (_abi.MESHES_V, _abi.MESHES_V_OLD, _abi.MESHES_VT),
                          (_abi.MESHES_W, _abi.MESHES_W_OLD, _abi.MESHES_WT),
                          (_abi.MESHES_T, _abi.MESHES_T_OLD, _abi.MESHES_TT)), fields(cell)):
            for f in fs:
                solver.upload(f, v)
    solver.add_temperature_noise(amp, seed)


class _Run:
    """One enclosure in a host program's hands: its solver, the restart
    arrays it starts from (page-locked, as a restart file is read) and the
    page-locked buffer its results land in."""

    def __init__(self, mp, params, roll, seed):
        self.mesh = nimgpu.Mesh(mp)
        self.solver = nimgpu.NimSolver(self.mesh, params)
        _start(self.solver, mp, roll, 1e-6, seed)
        self.fields = FACE_FIELDS + CELL_FIELDS + AVERAGES
        # one step, so that the arrays are those of a running program
        self.solver.solve_nse(1)
        sizes = [self.mesh.nface] * len(FACE_FIELDS) + [self.mesh.nmesh] * (len(CELL_FIELDS) + len(AVERAGES))
        self.start = torch.empty(sum(sizes), dtype=torch.float64, pin_memory=True).numpy()
        self.parts = np.split(self.start, np.cumsum(sizes)[:-1])
        for f, part in zip(self.fields, self.parts):
            self.solver.download(f, part)
        out = self.solver.output_array(_abi.OUTPUT_RESTART)
        self.out = torch.empty(out.size, dtype=torch.float64, pin_memory=True).numpy()

    def restart(self):
        for f, part in zip(self.fields, self.parts):
            self.solver.upload(f, part)

    def begin_output(self):
        return self.solver.output_begin(_abi.OUTPUT_RESTART, self.out)


def prepare(case, seed):
    if case["kind"] == "batch":
        runs = []
        for c in config.batch_cases(case["n"], seed=case["batch_seed"], a_min=case["a_min"], a_max=case["a_max"]):
            prec = _abi.PRECISION_MIXED if case["precision"] == "mixed" else _abi.PRECISION_FP64
            runs.append(_Run(c.mesh_params(), c.params(precision=prec), 0.0, c.seed + 1000 * seed))
        return {"case": case, "runs": runs}
    mp, params = _case_of(case)
    return {"case": case, "runs": [_Run(mp, params, case["roll"], seed)]}


def _records(recs):
    return {"iters": [r.iters for r in recs], "nu": np.array([[r.nu_inner, r.nu_outer] for r in recs]),
            "dilatation": np.array([r.dilatation for r in recs])}


def run(state):
    case, runs = state["case"], state["runs"]
    if case["kind"] == "tangent":
        s = runs[0].solver
        runs[0].restart()
        s.tangent_begin()
        s.tangent_seed(*s.tangent_seed_of("Ra", case["Ra"], case["Pr"]))
        recs, dnu = s.tangent_step(case["steps"])
        T, dT = s.tangent_get(_abi.MESHES_T)
        w, dw = s.tangent_get(_abi.FACES_W)
        return {**_records(recs), "dnu": dnu, "T": T, "dT": dT, "w": w, "dw": dw}
    for r in runs:
        r.restart()
    if case["kind"] == "batch":
        recs = nimgpu.batch_step([r.solver for r in runs], case["steps"], fused=case["form"] == "fused")
    else:
        recs = [runs[0].solver.solve_nse(case["steps"])]
    tickets = [r.begin_output() for r in runs]
    for r, t in zip(runs, tickets):
        r.solver.output_wait(t)
    return {"records": [_records(x) for x in recs], "restart": [r.out for r in runs]}


# Values a pass of the inner iteration cannot do without, per cell.  Read: the
# three faces a cell owns of u, v, w, p, T (15), its averages and old values
# (8), face areas and normals (12), volume (1), G (3), g^ij (9), xi_x (9), the
# diagonal and the differences of the face metric (12), the step's velocity
# NIM constants M_F4 (8) and M_F1..3 (15).  Written: the faces (15) and the
# averages (4).  Their number of passes is the case's, to a few per cent.
VALUES_PER_CELL = 111
# floating-point operations of a pass per cell: the sums of the gradients,
# metric products and NIM terms, and the temperature's NIM coefficients
FLOPS_PER_CELL = 2000


def work(case):
    if case["kind"] == "batch":
        cells = sum(c.ncells for c in config.batch_cases(case["n"], seed=case["batch_seed"], a_min=case["a_min"],
                                                         a_max=case["a_max"]))
    else:
        cells = case["n_theta"] * case["n_r"] * case["n_z"]
    width = 4 if case["precision"] == "mixed" else 16 if case["kind"] == "tangent" else 8
    passes = case["passes"] * case["steps"]
    state = 2 * 42 * 8  # the restart arrays in and out
    return {"bytes": float(cells) * (VALUES_PER_CELL * width * passes + state),
            "flops": float(cells) * FLOPS_PER_CELL * passes}


def exact(case, seed):
    """None: a time step's fields are the iterate at which the reference's
    stop test first holds, which has no value apart from that iteration in
    its own operation order (the FP64 path is defined to its last bit)."""
    return None
