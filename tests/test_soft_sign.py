"""Zero products of the integer path take the sign of both operands.

Every exponent a factor's record accepts, those it refuses, zero factors, and
either sign of the zero and of the factor; compared bit for bit with the
host's own products.
"""
import ctypes
import math
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_zero_products_keep_their_sign():
    out = HERE / "_build"
    out.mkdir(exist_ok=True)
    lib = out / "libsoft_sign.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(lib), str(HERE / "soft_sign_check.cpp")],
                   check=True)
    f = ctypes.CDLL(str(lib)).zero_times
    f.restype, f.argtypes = ctypes.c_double, [ctypes.c_double] * 2
    sizes = [m * 2.0 ** e for e in range(-140, 140) for m in (1.0, 1.37)] + [0.0, 5e-324, 1e300]
    for size in sizes:
        for c in (size, -size):
            for zero in (0.0, -0.0):
                assert math.copysign(1.0, f(zero, c)) == math.copysign(1.0, zero * c), (zero, c)
