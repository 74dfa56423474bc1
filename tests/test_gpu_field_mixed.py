"""Shortcuts of the mixed-precision field driver (gbx/FieldMixed.hh, GPU).

Each must give what the operations it stands for give: 1 / sqrt(x) for every
float of two binades (at the ends of its range and around 1), the acceptance
of a step and the FP32 error norm for errors around the acceptance limit, far
from it, zero and non-finite, and the conversions between FP32 and FP64 over
the whole range of positive numbers.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "field_mixed_eval.cu")
N = 1 << 18


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from celeritas_gb300.build import common_flags, nvcc_path

    out = str(tmp_path_factory.mktemp("field") / "libfield.so")
    subprocess.run([nvcc_path()] + common_flags("mixed") + ["-shared", "-o", out, SRC, "-lcudart"],
                   check=True, capture_output=True)
    return ctypes.CDLL(out)


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("exponent", [-75, -1, 0, 118])
def test_inverse_square_root(lib, exponent):
    bad = ctypes.c_uint(1)
    assert lib.inv_sqrt_mismatches(exponent, ctypes.byref(bad)) == 0
    assert bad.value == 0


@pytest.mark.parametrize("epsilon", [1e-3, 1e-5])
def test_error_norm(lib, epsilon):
    rng = np.random.default_rng(3)
    # Position error rate and relative momentum error around epsilon
    scale = epsilon * 10.0 ** np.where(rng.integers(0, 2, (N, 2)) == 0,
                                       rng.uniform(-1e-6, 1e-6, (N, 2)), rng.uniform(-9, 9, (N, 2)))
    unit = rng.normal(size=(3, N, 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    momentum = unit[2] * 10.0 ** rng.uniform(-4, 6, (N, 1))
    v = np.concatenate([unit[0] * scale[:, :1],
                        unit[1] * scale[:, 1:] * np.linalg.norm(momentum, axis=1, keepdims=True),
                        momentum], axis=1).astype(np.float32)
    v[:8, :6] = 0
    v[8:16, 0] = np.inf
    v[16:24, 4] = np.nan
    v[24:32, 6:] = 0
    out = np.empty((N, 4), np.float32)
    assert lib.error_norms(ctypes.c_double(epsilon), ptr(v), ptr(out), N) == 0
    np.testing.assert_array_equal(out[:, 0], out[:, 1])
    np.testing.assert_array_equal(out[:, 2], out[:, 3])


def test_conversions(lib):
    rng = np.random.default_rng(4)
    d = 10.0 ** rng.uniform(-60, 60, N)
    d[:N // 2] = np.abs(rng.integers(1, 0x7f000000, N // 2).astype(np.int32).view(np.float32)
                        .astype(float)) * (1 + rng.integers(-3, 4, N // 2) * 2.0**-25)
    d[:6] = [0.0, np.inf, 1e-46, 3.4028235677973366e38, 1.1754943508222875e-38, 2.0**-149]
    f = rng.integers(0, 0x7f800001, N).astype(np.uint32).view(np.float32).copy()
    to, back = np.empty(N, np.float32), np.empty(N)
    assert lib.conversions(ptr(d), ptr(f), ptr(to), ptr(back), N) == 0
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(to, d.astype(np.float32))
    np.testing.assert_array_equal(back, f.astype(float))
