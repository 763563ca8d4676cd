"""gm_moved_far (csrc/gm_exact_math.h), compiled as C11: never false for a squared
displacement at or past the threshold, false only below it, and true for a NaN
of either sign (the GPU's own NaN has the sign bit set)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = """
#include "gm_exact_math.h"
void far_of(long n, const double *d2, double far_sq, int *out) {
    for (long i = 0; i < n; i++) out[i] = gm_moved_far(d2[i], far_sq);
}
"""


@pytest.fixture(scope="module")
def far(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("moved_far")
    src, lib = tmp / "m.c", tmp / "m.so"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(HERE), "geodesic-m_gb300", "csrc")
    subprocess.check_call(["gcc", "-std=c11", "-O2", "-shared", "-fPIC", "-I", inc, str(src), "-o", str(lib), "-lm"])
    L = ctypes.CDLL(str(lib))

    def call(d2, t):
        d2 = np.ascontiguousarray(d2, np.float64)
        out = np.empty(len(d2), np.int32)
        L.far_of(ctypes.c_long(len(d2)), d2.ctypes.data_as(ctypes.c_void_p), ctypes.c_double(t),
                 out.ctypes.data_as(ctypes.c_void_p))
        return out
    return call


@pytest.mark.parametrize("t", [0.0, 1e-6, 0.249001, 0.25, 1.0, 6.2])
def test_threshold(far, t):
    r = np.random.default_rng(1)
    d2 = np.concatenate([r.uniform(0, 3 * t, 100_000), t * (1 + np.arange(-40, 41) * 2.0 ** -52),
                         t * (1 + np.arange(-40, 41) * 2.0 ** -20), [0.0, 1e300, np.inf]])
    f = far(d2, t)
    assert np.all(f[d2 >= t] == 1)
    assert np.all(d2[f == 1] >= t * (1 - 2.0 ** -20))  # the high word's resolution


def test_nan_of_either_sign(far):
    nan = np.array([0x7ff8000000000000, 0xfff8000000000000, 0x7ff0000000000001, 0xffffffffffffffff], np.uint64)
    assert np.all(far(nan.view(np.float64), 0.25) == 1)
