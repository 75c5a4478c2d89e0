"""The shared-divisor quotients of the device models (models.cuh Divisor):
with r = 1 / b rounded to nearest, q0 = a r and two corrections by the exact
residual, q + (a - q b) r, round as the division does. Restated here with the
C library's fma; random operands and the mantissas where a rounding could
slip (all ones, one bit off a power of two, neighbours of each other). And
the device code itself (divisor_probe.cu), with every kind of operand it
sends to the division instead."""

import ctypes
import ctypes.util
import math
import os
import random
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

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


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("divisor") / "probe.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O2", "--fmad=false", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(ROOT, "espice_b200", "csrc"), os.path.join(ROOT, "tests", "divisor_probe.cu"), "-o",
                    so], check=True)
    return ctypes.CDLL(so).probe


def edges():
    """Zeros, infinities, NaN, subnormals, and the neighbours of the ends of
    the range that takes the shared reciprocal (2^-511, 2^511), of the normal
    numbers and of 1, each sign."""
    out = [0.0, math.inf, math.nan, 5e-324, 1e-310]
    for e in (-1022, -1021, -512, -511, -510, -1, 0, 1, 509, 510, 511, 512, 1023):
        x = math.ldexp(1.0, e)
        out += [x, math.nextafter(x, 0.0), math.nextafter(x, math.inf), x * (2.0 - 2.0 ** -52)]
    return np.array(out + [-x for x in out])


@pytest.mark.gpu
@pytest.mark.parametrize("kinds", ["edges", "random", "ones", "low", "sparse"])
def test_device_quotients_are_the_divisions(probe, kinds):
    import torch
    if kinds == "edges":
        e = edges()
        a, b = (x.ravel() for x in np.meshgrid(e, e))
    else:
        rng = random.Random(kinds)
        a, b = (np.array([operand(rng, k) for _ in range(1 << 17)]) for k in (kinds, rng.choice(["random", "ones"])))
    n = len(a)
    da, db = torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")
    one, three, div = (torch.zeros(k * n, dtype=torch.float64, device="cuda") for k in (1, 3, 3))
    torch.cuda.synchronize()
    assert probe(*[ctypes.c_void_p(t.data_ptr()) for t in (da, db, one, three, div)], n) == 0
    one, three, div = (t.cpu().numpy() for t in (one, three, div))
    with np.errstate(all="ignore"):
        host = a / b
    for got, want in ((div[:n], host), (one, div[:n]), (three, div)):
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))
