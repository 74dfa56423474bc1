"""Errors of the fixed-point elementary functions (gbx/LibmInt.hh) before rounding.

A result is rounded when the error allowed for it cannot change the rounding, so every
result's error has to stay below that one, with a margin: the worst cases of the
truncations sum to at most 0.65 of it, and no argument may exceed three quarters. Arguments
are random over the range covered, and dense where the error is largest: |log| just below
2^-7, pi/4, 0.35 and the halves of ln 2 / 128.
"""

import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "libm_int_eval.cc")
N = 8000
FUNCTIONS = ("exp", "log", "sin", "cos", "expm1", "log1p")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("libm") / "libmargin.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", out,
                    SRC], check=True)
    return ctypes.CDLL(out)


def arguments(fn, rng):
    sign = rng.choice([-1.0, 1.0], N)
    near = 1 - 2.0 ** rng.uniform(-20, -4, N)  # just below one
    if fn == "exp":
        half = (rng.integers(0, 130000, N) + 0.5) * math.log(2) / 128
        return np.concatenate([sign * rng.uniform(0, 708, N), sign * half,
                               sign * 2.0 ** rng.uniform(-53, 9, N)])
    if fn == "log":
        return np.concatenate([1 + 2.0**-7 * near, 1 - 2.0**-8 * near, rng.uniform(0.5, 2, N),
                               2.0 ** rng.uniform(-1000, 1000, N)])
    if fn == "log1p":
        return np.concatenate([sign * 2.0**-7 * near, sign * 2.0 ** rng.uniform(-53, -7.01, N),
                               -rng.uniform(2.0**-7, 0.999, N)])
    if fn == "expm1":
        return np.concatenate([sign * 0.3499 * near, sign * rng.uniform(0.001, 0.3499, N),
                               sign * 2.0 ** rng.uniform(-53, -2, N)])
    octant = rng.integers(1, 1300, N) * (math.pi / 4) * near
    return np.concatenate([sign * rng.uniform(0, 1023, N), sign * octant,
                           sign * 2.0 ** rng.uniform(-25, 9, N)])


@pytest.mark.parametrize("fn", FUNCTIONS)
def test_error_is_below_the_allowed_one(lib, fn):
    x = arguments(fn, np.random.default_rng(FUNCTIONS.index(fn)))
    hi, lo = np.empty(len(x), np.uint64), np.empty(len(x), np.uint64)
    e, bits = np.empty(len(x), np.int32), np.empty(len(x), np.int32)
    lib.libm_unrounded(FUNCTIONS.index(fn), *(a.ctypes.data_as(ctypes.c_void_p)
                                              for a in (x, hi, lo, e, bits)), len(x))
    assert np.mean(bits != 0) > 0.99
    with mpmath.workprec(200):
        f, worst = getattr(mpmath, fn), 0.0
        for i in np.flatnonzero(bits):
            v = mpmath.ldexp((int(hi[i]) << 64) + int(lo[i]), int(e[i]) - 127)
            error = abs(v - abs(f(mpmath.mpf(float(x[i])))))
            worst = max(worst, float(mpmath.ldexp(error, int(bits[i]) - int(e[i]))))
    assert worst < 0.75
