"""The form the reference order's sweeps take on a mesh (nim_reference_form,
include/nim_gpu.h): skewed copies only where they stay a small multiple of
the fields or a few GB, and their planes can be indexed in 32 bits.  Pure host functions
of libnimgpu.so: no GPU needed."""
import ctypes as C
import random

import numpy as np
import pytest

from nimgpu import _abi

SHARED, GRID, SKEWED = 0, 1, 2
PLANES = 27  # three components of 6 planes, the pressure's 4, the temperature's 5
LIMIT = 4 << 30  # bytes of copies that outgrow 8 values a cell and plane


@pytest.fixture(scope="module", autouse=True)
def gpu_lib():
    if not _abi.gpu_lib_path().exists():
        pytest.skip("libnimgpu.so not built (needs nvcc: __graft_entry__.build())")


def form(nt, nr, nz):
    copies = C.c_int64(-1)
    return _abi.gpu_lib().nim_reference_form(nt, nr, nz, C.byref(copies)), copies.value


def plane(nt, nr, nz):  # values of a skewed plane, in Python's integers
    levels = (nt - 1) + 2 * (nr - 1) + 3 * (nz - 1) + 1
    return (levels + 3) * (nz + 1) * (nr + 1)


def widest_level(nt, nr, nz):
    step = np.zeros(nt + 2 * nr + 3 * nz, dtype=np.int64)
    j, k = np.meshgrid(np.arange(nr), np.arange(nz), indexing="ij")
    np.add.at(step, (2 * j + 3 * k).ravel(), 1)
    np.add.at(step, (2 * j + 3 * k + nt).ravel(), -1)
    return int(np.cumsum(step).max())


# tall, deep and long meshes of narrow levels: the planes outgrow the mesh, or
# 32 bits, or both (36x80x4300 wraps to a small positive number, 24x120x2500
# to a negative one, and 6x10x11410 to one smaller than the mesh)
@pytest.mark.parametrize("dims", [(36, 80, 400), (36, 80, 2000), (36, 80, 4300), (24, 120, 2500), (6, 480, 2000),
                                  (6, 10, 11410), (12, 60, 800), (12, 128, 2000), (24, 24, 600)])
def test_narrow_levels_of_a_stretched_mesh_sweep_the_fields(dims):
    assert widest_level(*dims) <= 1024
    assert plane(*dims) > 8 * np.prod(dims, dtype=np.int64) and 8 * PLANES * plane(*dims) > LIMIT
    assert form(*dims) == (GRID, 0)


@pytest.mark.parametrize("dims,want", [
    ((36, 6, 12), SHARED), ((36, 14, 13), SHARED), ((36, 14, 14), SKEWED), ((24, 24, 16), SKEWED),
    ((48, 48, 32), SKEWED), ((60, 40, 30), SKEWED), ((301, 5, 6), SKEWED), ((24, 24, 200), SKEWED), ((16, 60, 300), SKEWED),
    ((6, 10, 600), SKEWED), ((90, 70, 60), GRID), ((128, 128, 96), GRID)])
def test_the_measured_meshes_keep_their_form(dims, want):
    got, copies = form(*dims)
    assert got == want
    assert copies == (8 * PLANES * plane(*dims) if want == SKEWED else 0)


def test_skewed_copies_stay_small_and_inside_32_bits():
    rng = random.Random(5)
    seen = {SHARED: 0, GRID: 0, SKEWED: 0}
    for _ in range(4000):
        nt = round(6 * 10 ** rng.uniform(0, rng.choice((1, 2, 5))))
        nr = round(3 * 10 ** rng.uniform(0, 2.5))
        nz = round(3 * 10 ** rng.uniform(0, 3))
        if nt * nr * nz > (2 ** 31 - 1) // 20:
            continue
        got, copies = form(nt, nr, nz)
        seen[got] += 1
        if widest_level(nt, nr, nz) > 1024:
            assert got == GRID
        if got == SKEWED:
            n = plane(nt, nr, nz)
            assert copies == 8 * PLANES * n <= max(8 * PLANES * 8 * nt * nr * nz, LIMIT)
            # the largest index of a sweep: three planes and the farthest neighbour
            assert 3 * n + 8 * (nz + 1) * (nr + 1) < 2 ** 31
        else:
            assert copies == 0
    assert min(seen.values()) > 100


@pytest.mark.parametrize("dims", [(5, 3, 3), (6, 2, 3), (6, 3, 2), (-6, 3, 3), (2 ** 15, 2 ** 15, 3)])
def test_counts_create_refuses(dims):
    assert form(*dims)[0] == _abi.NIM_ERR_BAD_ARG
