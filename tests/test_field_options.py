"""The mixed field driver's error norm for any tolerance (no GPU).

Its FP32-pair form must decide and round as FP64 does for every 'epsilon_rel_max' that is
accepted, also where its square's reciprocal, which the pairs are multiplied by, leaves the
range in which two FP32 numbers hold it.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "field_options_eval.cc")
N = 1 << 15


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("field") / "libfieldopt.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    "-DGBX_PHYS_REAL=float", "-o", out, SRC], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("epsilon", [1e-170, 1e-30, 1e-15, 1e-3, 1.0, 1e10, 1e14, 1e16, 1e18,
                                     1e19, 3e19, 1e20, 1e22, 1e25, 1e160])
def test_error_norm(lib, epsilon):
    rng = np.random.default_rng(8)
    # Errors whose squares span the range that the pairs are used in, and around epsilon
    scale = 10.0 ** rng.uniform(-9, 9, (N, 2))
    near = epsilon * 10.0 ** rng.uniform(-1e-6, 1e-6, (N, 2))
    scale = np.where((rng.integers(0, 4, (N, 2)) == 0) & (near > 1e-9) & (near < 1e9), near, scale)
    unit = rng.normal(size=(3, N, 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    momentum = unit[2] * 10.0 ** rng.uniform(-2, 5, (N, 1))
    v = np.concatenate([unit[0] * scale[:, :1],
                        unit[1] * scale[:, 1:] * np.linalg.norm(momentum, axis=1, keepdims=True),
                        momentum], axis=1).astype(np.float32)
    out = np.empty((N, 4), np.float32)
    lib.error_norms(ctypes.c_double(epsilon), v.ctypes.data_as(ctypes.c_void_p),
                    out.ctypes.data_as(ctypes.c_void_p), N)
    np.testing.assert_array_equal(out[:, 0], out[:, 1])
    np.testing.assert_array_equal(out[:, 2], out[:, 3])
