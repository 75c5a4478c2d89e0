"""The shared-divisor quotients of the device models (models.cuh Divisor):
with r = 1 / b rounded to nearest, q0 = a r and two corrections by the exact
residual, q + (a - q b) r, round as the division does. Restated here with the
C library's fma; random operands and the mantissas where a rounding could
slip (all ones, one bit off a power of two, neighbours of each other)."""

import ctypes
import ctypes.util
import math
import random

import pytest

_libm = ctypes.CDLL(ctypes.util.find_library("m"))
_libm.fma.restype = ctypes.c_double
_libm.fma.argtypes = [ctypes.c_double] * 3
fma = _libm.fma


def quotient(a, b):
    r = 1.0 / b
    q = a * r
    for _ in range(2):
        q = fma(fma(-b, q, a), r, q)
    return q


def operand(rng, kind):
    m = {"random": rng.getrandbits(52), "ones": (1 << 52) - 1 - rng.randrange(3), "low": rng.randrange(4),
         "sparse": (1 << rng.randrange(52)) | (1 << rng.randrange(52))}[kind]
    return math.ldexp(1.0 + m / (1 << 52), rng.randrange(-510, 511)) * rng.choice((-1.0, 1.0))


@pytest.mark.parametrize("ka", ["random", "ones", "low", "sparse"])
@pytest.mark.parametrize("kb", ["random", "ones", "low", "sparse"])
def test_quotients_round_as_the_division(ka, kb):
    rng = random.Random(f"{ka}/{kb}")
    for _ in range(4000):
        a, b = operand(rng, ka), operand(rng, kb)
        assert quotient(a, b) == a / b, (a.hex(), b.hex())
