"""Zero numerators of the straight-line quotients (csrc/nim_div.cuh) keep the
sign the host's division gives them."""
import ctypes as C

import numpy as np
import pytest

from nimgpu import _abi

pytestmark = pytest.mark.gpu


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def test_zero_numerators_keep_their_sign():
    b = np.array([1.0, -1.0, 3.0, -3.0, 2.0 ** 400, -(2.0 ** -400), 1.75, 2 - 2.0 ** -30, -np.inf, np.inf])
    a = np.concatenate([np.zeros(b.size), -np.zeros(b.size)])
    b = np.tile(b, 2)
    q = np.empty_like(a)
    assert _abi.gpu_lib().nim_gpu_selftest_quot(ptr(a), ptr(b), ptr(q), a.size) == _abi.NIM_OK
    assert np.array_equal(q.view(np.int64), (a / b).view(np.int64))

