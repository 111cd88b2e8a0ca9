"""The mixed hat pass's sums of squares (csrc/fx_weight.cuh, Squares), compiled for the host, against exact sums.

The bar is 2^-27 of the sum, well below the 2^-23 that the rounding of a float is of its square, for values of any
magnitude (absolutely 8 x 2^-93 where nothing is above 2^-33); in the pass a sum spans up to 64 values, 2^-40."""
import ctypes
import os
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sq") / "fx_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "arith", "fx_host.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.fx_squares.restype = ctypes.c_double
    lib.fx_squares.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_double]
    return lib


@pytest.mark.parametrize("low,high", [(0, 0), (-8, 0), (-17, -15), (-30, 0), (-31, -20), (-40, -30), (-60, -40), (-100, 0)])
def test_sums(host, low, high):
    rng = random.Random(low * 7 + high)
    for _ in range(400):
        n = rng.randint(1, 8)
        s = np.array([rng.choice([-1, 1]) * rng.random() * 2.0 ** rng.uniform(low, high) for _ in range(n)], np.float32)
        want = sum(Fraction(float(v)) ** 2 for v in s)
        got = Fraction(host.fx_squares(s.ctypes.data, n, 0.0))
        assert abs(got - want) <= want * Fraction(1, 2 ** 27) + Fraction(8, 2 ** 93), (s, float(got), float(want))


def test_a_pass_long(host):
    rng = np.random.default_rng(1)
    for low in (-1, -20, -40):
        s = (rng.standard_normal(64) * 2.0 ** low).astype(np.float32)
        want = sum(Fraction(float(v)) ** 2 for v in s)
        assert abs(Fraction(host.fx_squares(s.ctypes.data, 64, 0.0)) - want) <= want * Fraction(1, 2 ** 40)


def test_edges(host):
    for v in (0.0, -0.0, 1.0 - 2.0 ** -24, 2.0 ** -16, -(2.0 ** -16), np.nextafter(np.float32(2.0 ** -16), np.float32(0))):
        s = np.full(8, v, np.float32)
        want = 8 * Fraction(float(s[0])) ** 2
        assert abs(Fraction(host.fx_squares(s.ctypes.data, 8, 0.0)) - want) <= want * Fraction(1, 2 ** 27)
