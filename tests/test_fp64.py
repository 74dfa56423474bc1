"""FP64 division, square root (gbx/Fp64.hh) and elementary functions
(gbx/LibmInt.hh) in integer arithmetic.

The first two are IEEE operations rounded to nearest even, so every result must equal
numpy's bit for bit. The operands cover the edges of the significand (all
zeros, all ones, short and long runs of either), of the exponent range (the
last normal and subnormal results, overflow) and the special values. The
significand routines are also run on the host with the FP32 approximation
they start from moved by 3 units in its last place, more than the 1 (rcp) and
2 (rsqrt) that the hardware's instructions document. The elementary functions
must return the correctly rounded value wherever they decide one, and decide
all but a few in 2^9 arguments of the range they cover, to its edges.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fp64_eval.cu")
N = 1 << 18
MASK = (1 << 52) - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from celeritas_gb300.build import common_flags, nvcc_path

    out = str(tmp_path_factory.mktemp("fp64") / "libfp64.so")
    subprocess.run([nvcc_path()] + common_flags() + ["-shared", "-o", out, SRC, "-lcudart"],
                   check=True, capture_output=True)
    return ctypes.CDLL(out)


def significands(rng, n):
    """53-bit significands: random ones and the edges of the range."""
    m = rng.integers(0, MASK + 1, n, dtype=np.uint64)
    kind = rng.integers(0, 6, n)
    shift = rng.integers(1, 52, n).astype(np.uint64)
    ones = (np.uint64(1) << shift) - np.uint64(1)
    m = np.where(kind == 0, m & np.uint64(15), m)
    m = np.where(kind == 1, np.uint64(MASK) - (m & np.uint64(15)), m)
    m = np.where(kind == 2, m & ~ones, m)
    m = np.where(kind == 3, m | ones, m)
    return (m & np.uint64(MASK)) | np.uint64(1 << 52)


def fractions(y):
    return (y.view(np.uint64) & np.uint64(MASK)) | np.uint64(1 << 52)


@pytest.mark.parametrize("ulps", [-3, 0, 3])
def test_significands(lib, ulps):
    rng = np.random.default_rng(17 + ulps)
    a, b, y = significands(rng, N), significands(rng, N), np.empty(N, np.uint64)

    def evaluate(op, x):
        lib.fp64_host(op, x.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                      y.ctypes.data_as(ctypes.c_void_p), N, ulps)
        return y

    np.testing.assert_array_equal(evaluate(0, a), fractions(a.astype(float) / b.astype(float)))
    x = a << rng.integers(0, 2, N).astype(np.uint64)
    root = np.sqrt(x.astype(float) * 2.0**-52)
    expected = np.where(root < 2, fractions(root), np.uint64(1 << 53))
    np.testing.assert_array_equal(evaluate(1, x), expected)


#: Range that the fixed-point functions cover, by magnitude and sign
COVERED = {"exp": (2.0**-54, 708.3), "log": (2.3e-308, 1.7e308), "sin": (2.0**-26, 1023.9),
           "cos": (2.0**-26, 1023.9), "expm1": (2.0**-54, 0.3499), "log1p": (2.0**-54, 0.9999)}


@pytest.mark.parametrize("fn", list(COVERED))
def test_fixed_point_functions(lib, built_port, fn):
    import oracle

    rng = np.random.default_rng(list(COVERED).index(fn))
    lo, hi = COVERED[fn]
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), N))
    x[:N // 2] = rng.uniform(lo, min(hi, 50.0), N // 2)
    if fn == "log":
        # Around 1, and the intervals that meet there
        x[:N // 8] = 1 + rng.uniform(-1, 1, N // 8) * 2.0 ** rng.uniform(-40, -5, N // 8)
    else:
        x *= rng.choice([-1.0, 1.0], N)
    if fn == "log1p":
        x = np.where((x > 0) & (x >= 2.0**-7), -x, x)
    y, decided = np.empty(N), np.empty(N, np.uint8)
    lib.libm_fixed(list(COVERED).index(fn), x.ctypes.data_as(ctypes.c_void_p),
                   y.ctypes.data_as(ctypes.c_void_p),
                   decided.ctypes.data_as(ctypes.c_void_p), N)
    ok = decided != 0
    expected = oracle.port_libm(fn, x)
    np.testing.assert_array_equal(y[ok].view(np.uint64), expected[ok].view(np.uint64))
    # Tiny arguments (results near 1 or near the argument) are left out more
    # often: a midpoint lies at half the last place of either
    usual = (np.abs(x - (fn == "log")) > 2.0**-20)
    assert np.mean(~ok[usual]) < 2.0**-8


@pytest.mark.gpu
def test_device_matches_ieee(lib):
    rng = np.random.default_rng(5)

    def operands(special):
        e = rng.integers(0, 2048, N)
        near = rng.integers(0, 2, N) == 0
        e = np.where(near, rng.integers(1023 - 40, 1023 + 40, N), e).astype(np.uint64)
        sign = rng.integers(0, 2, N).astype(np.uint64) << np.uint64(63)
        x = (sign | (e << np.uint64(52)) | (significands(rng, N) & np.uint64(MASK))).view(float)
        x[:len(special)] = special
        return x

    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072014e-308,
                        1.7976931348623157e308, 1.0, -1.0])
    a = operands(np.repeat(special, len(special)))
    b, y = operands(np.tile(special, len(special))), np.empty(N)
    with np.errstate(all="ignore"):
        for op, expected in ((0, a / b), (1, np.sqrt(a))):
            rc = lib.fp64_device(op, a.ctypes.data_as(ctypes.c_void_p),
                                 b.ctypes.data_as(ctypes.c_void_p),
                                 y.ctypes.data_as(ctypes.c_void_p), N)
            assert rc == 0
            np.testing.assert_array_equal(np.isnan(y), np.isnan(expected))
            ok = ~np.isnan(expected)
            np.testing.assert_array_equal(y[ok].view(np.uint64), expected[ok].view(np.uint64))
