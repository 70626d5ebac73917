"""The straight-line quotients of the FP64 sweeps (csrc/nim_div.cuh) and the
NIM coefficients built on them, bit for bit: a / b as the host's IEEE
division rounds it, and nim_direction as nim.f90:181-287 evaluates it (host
double arithmetic and libm exp) on both sides of every branch: the series
that stops at its last effective term, the full one beyond |Re| = 0.01, the
exponential form, and operands only the general form takes."""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import pytest

from nimgpu import _abi

pytestmark = pytest.mark.gpu


def ptr(a: np.ndarray):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def quot(a: np.ndarray, b: np.ndarray) -> np.ndarray:
    a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
    q = np.empty_like(a)
    assert _abi.gpu_lib().nim_gpu_selftest_quot(ptr(a), ptr(b), ptr(q), a.size) == _abi.NIM_OK
    return q


def same(x, y):
    x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
    eq = (x.view(np.int64) == y.view(np.int64)) | ((x == 0) & (y == 0)) | (np.isnan(x) & np.isnan(y))
    return eq


def operands(kind: str):
    rng = np.random.default_rng(17)
    n = 4_000_000
    ma, mb = rng.uniform(1, 2, n), rng.uniform(1, 2, n)
    sign = rng.choice((-1.0, 1.0), n)
    if kind == "near one exponent":
        return sign * ma, mb
    if kind == "the whole range":
        return sign * np.ldexp(ma, rng.integers(-479, 480, n)), np.ldexp(mb, rng.integers(-479, 480, n))
    if kind == "divisors just below two":  # both sides of the accepted significands
        return ma, np.ldexp(2.0 - np.ldexp(rng.uniform(0, 4, n), -rng.integers(19, 53, n)), rng.integers(-9, 9, n))
    if kind == "quotients next to a midpoint":  # a = the double nearest (q + half an ulp) b
        mb, q = mb[:200_000], ma[:200_000]
        a = [float((Fraction(x) + Fraction(1, 2 ** 53)) * Fraction(y)) for x, y in zip(q, mb)]
        a = np.array(a)
        return np.concatenate([a, np.nextafter(a, 0), np.nextafter(a, 4)]), np.tile(mb, 3)
    special = np.array([0.0, -0.0, 1.0, -1.0, 2.0 ** -1074, 2.0 ** -500, 2.0 ** 500, 1.7e308, np.inf, -np.inf, np.nan,
                        2 - 2.0 ** -52, 1 + 2.0 ** -52, 3.0, 1 / 3])
    return np.repeat(special, special.size), np.tile(special, special.size)


@pytest.mark.parametrize("kind", ["near one exponent", "the whole range", "divisors just below two",
                                  "quotients next to a midpoint", "special values"])
def test_quotients_are_correctly_rounded(kind):
    a, b = operands(kind)
    with np.errstate(all="ignore"):
        want = a / b
    eq = same(quot(a, b), want)
    assert eq.all(), (a[~eq][:3], b[~eq][:3])


def powers(x):
    p = [1.0, x, x * x]
    p.append(p[1] * p[2])
    p.append(p[2] * p[2])
    p.append(p[2] * p[3])
    p.append(p[3] * p[3])
    p.append(p[3] * p[4])
    p.append(p[4] * p[4])
    p.append(p[3] * p[6])
    p.append(p[5] * p[5])
    p.append(p[5] * p[6])
    return p


def reference(u, k, v_limit):
    """nim.f90:181-287 for one direction, a = gminus = gplus = 1."""
    Re = 2 * u / k
    if abs(Re) > v_limit:
        e = math.exp(Re)
        A = [2 / (k * (1 / e - 1)) + 1 / u, -(2 / (k * (1 - e))) - 1 / u, u / (k * (1 / e - 1)), u / (k * (1 - e))]
        if Re > 0:
            return A + [(-k + u * (1 / e + 1) / (-(1 / e) + 1)) / (u * u), 1 / (-(1 / e) + 1) - 1 / Re]
        return A + [(-k + u * (1 + e) / (-1 + e)) / (u * u), e / (-1 + e) - 1 / Re]
    U, K = powers(u), powers(k)
    s1 = [u / (3 * K[2]), U[3] / (45 * K[4]), 2 * U[5] / (945 * K[6]), U[7] / (4725 * K[8]), 2 * U[9] / (93555 * K[10])]
    s2 = [U[2] / (6 * K[2]), U[4] / (90 * K[4]), U[6] / (945 * K[6]), U[8] / (9450 * K[8]), U[10] / (93555 * K[10])]
    return [-(1 / k) - s1[0] + s1[1] - s1[2] + -s1[3] - s1[4], -(1 / k) + s1[0] - s1[1] + s1[2] - -s1[3] + s1[4],
            -0.5 - u / (2 * k) - s2[0] + s2[1] - -s2[2] + s2[3] - s2[4],
            -0.5 + u / (2 * k) - s2[0] + s2[1] - -s2[2] + s2[3] - s2[4],
            1 / (3 * k) - U[2] / (45 * K[3]) + 2 * U[4] / (945 * K[5]) - -(U[6] / (4725 * K[7])) +
            2 * U[8] / (93555 * K[9]) - -(1382 * U[10] / (6.38512875e8 * K[11])),
            0.5 + u / (6 * k) - U[3] / (90 * K[3]) + U[5] / (945 * K[5]) - -(U[7] / (9450 * K[7])) + U[9] / (93555 * K[9])]


@pytest.mark.parametrize("lo,hi,v_limit", [
    (1e-12, 1e-4, 1e-2), (1e-4, 0.0101, 1e-2), (0.0099, 0.0101, 1e-2), (0.0101, 60.0, 1e-2), (150.0, 600.0, 1e-2),
    (1e-3, 0.3, 0.2),  # series beyond the trimmed range
    (1e-3, 0.3, 1e-3),  # exponential form inside it
])
def test_nim_coefficients_bit_for_bit(lo, hi, v_limit):
    rng = np.random.default_rng(29)
    n = 12_000
    k = 10.0 ** rng.uniform(-3, 5, n)
    Re = rng.choice((-1.0, 1.0), n) * np.exp(rng.uniform(math.log(lo), math.log(hi), n))
    u = Re * k / 2
    u[:3] = 0.0 if lo < v_limit else u[:3]
    A = np.empty(6 * n)
    assert _abi.gpu_lib().nim_gpu_selftest_nim_coef(ptr(u), ptr(k), n, _abi.PRECISION_FP64, v_limit, ptr(A)) == 0
    want = np.array([reference(float(x), float(y), v_limit) for x, y in zip(u, k)])
    eq = same(A.reshape(n, 6), want)
    assert eq.all(), (u[~eq.all(axis=1)][:3], k[~eq.all(axis=1)][:3])
