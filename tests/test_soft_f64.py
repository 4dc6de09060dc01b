"""The leapfrog's integer multiply and divide give the IEEE results.

CPU build of phonomena_gb300/csrc/soft_f64.cuh against the host's own FP64
operations, tolerance 0: random operands over the accepted exponent range,
short and long runs of ones and zeros in the significand, powers of two,
multiples of the divisor, and operands whose quotient or product lies next to
a rounding midpoint (or, for products, on it).
"""
import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def soft():
    out = HERE / "_build"
    out.mkdir(exist_ok=True)
    lib = out / "libsoft_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(lib),
                    str(HERE / "soft_check.cpp")], check=True)
    L = ctypes.CDLL(str(lib))
    L.soft_check.restype = ctypes.c_long
    L.soft_check.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_long] + [ctypes.POINTER(ctypes.c_long)] * 2
    return L


def significands(rng, n):
    """53-bit significands, a third of them with a long run of zeros or ones at the end."""
    m = rng.integers(1 << 52, 1 << 53, n, dtype=np.uint64)
    cut = (np.uint64(1) << rng.integers(1, 53, n, dtype=np.uint64)) - np.uint64(1)
    how = rng.integers(0, 6, n)
    m = np.where(how == 0, m & ~cut, np.where(how == 1, m | cut, m))
    return np.clip(m, 1 << 52, (1 << 53) - 1)


def numbers(rng, n, lo, hi):
    return np.ldexp(significands(rng, n).astype(np.float64), rng.integers(lo, hi, n) - 52) * rng.choice([-1.0, 1.0], n)


def near_midpoints(b, c):
    """x whose quotient by b, or product with c, is next to a midpoint of two doubles."""
    out = []
    mb, mc = int(math.frexp(b)[0] * 2 ** 53), int(abs(math.frexp(c)[0]) * 2 ** 53)
    for m in (mb, mc):
        odd = m >> ((m & -m).bit_length() - 1)
        inv = pow(odd, -1, 2 ** 54)
        for t in list(range(-24, 25)) + [2 ** 53 + t for t in range(-4, 5)]:  # odd * X = t (mod 2^54): product next to a midpoint
            x = (t * inv) % (2 ** 54)
            while x and x < 2 ** 52:
                x *= 2
            if 2 ** 52 <= x < 2 ** 53:
                out.append(float(x))
        for t in range(-24, 25):  # X * 2^54 = t (mod odd): quotient next to a midpoint
            x = (t * pow(2 ** 54, -1, odd)) % odd if odd > 1 else 0
            while x and x < 2 ** 52:
                x *= 2
            if 2 ** 52 <= x < 2 ** 53:
                out.append(float(x))
    return out


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("seed", range(4))
def test_integer_operations_equal_ieee(soft, kind, seed):
    rng = np.random.default_rng(seed)
    xs, bs, cs = [], [], []
    for b, c in zip(np.abs(numbers(rng, 300, -40, 40)), numbers(rng, 300, -120, 120)):
        if rng.random() < 0.1:
            b = 2.0 ** rng.integers(-40, 40)
        x = np.concatenate([numbers(rng, 2000, -720, 670), b * rng.integers(-500, 500, 200), [b, -b, 1.0 / b, 1.0],
                            np.multiply.outer(near_midpoints(b, c), [1.0, -2.0 ** -300, 2.0 ** 300]).ravel()])
        xs.append(x)
        bs.append(np.full(x.size, b))
        cs.append(np.full(x.size, c))
    x, b, c = (np.ascontiguousarray(np.concatenate(v)) for v in (xs, bs, cs))
    taken, exact = ctypes.c_long(), ctypes.c_long()
    bad = soft.soft_check(kind, x.ctypes.data, b.ctypes.data, c.ctypes.data, x.size, ctypes.byref(taken), ctypes.byref(exact))
    assert bad == 0
    assert taken.value > 0.9 * x.size and exact.value > 1000  # the exact path is exercised too


def test_operands_outside_the_range_are_refused(soft):
    """Zeros, subnormals, extremes, infinities and NaN are left to the FP64 operations."""
    x = np.array([0.0, -0.0, 5e-324, 1e-250, 1e250, np.inf, -np.inf, np.nan])
    one = np.ones_like(x)
    taken, exact = ctypes.c_long(), ctypes.c_long()
    assert soft.soft_check(0, x.ctypes.data, one.ctypes.data, one.ctypes.data, x.size, ctypes.byref(taken),
                           ctypes.byref(exact)) == 0
    assert taken.value == 0
    for b, c in ((-1.0, 0.0), (1e-60, -0.0), (1e60, 1e-60)):  # negative or extreme divisors, zero or extreme factors
        x, bb, cc = np.array([1.5]), np.array([b]), np.array([c])
        for kind in (0, 1):
            soft.soft_check(kind, x.ctypes.data, bb.ctypes.data, cc.ctypes.data, 1, ctypes.byref(taken), ctypes.byref(exact))
            assert taken.value == 0
