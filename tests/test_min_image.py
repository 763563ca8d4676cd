"""gm_min_image (csrc/gm_exact_math.h), compiled as C11 without contraction,
against the reference's expression d - L round(d / L) (neighbor.rs:74-76):
equal for every d, the boundaries of its three branches included."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = """
#include "gm_exact_math.h"
void images(long n, const double *d, double L, double *a, double *b) {
    for (long i = 0; i < n; i++) { a[i] = gm_min_image(d[i], L); b[i] = d[i] - L * round(d[i] / L); }
}
"""


@pytest.fixture(scope="module")
def images(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("min_image")
    src, lib = tmp / "m.c", tmp / "m.so"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(HERE), "geodesic-m_gb300", "csrc")
    subprocess.check_call(["gcc", "-std=c11", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc, str(src), "-o",
                           str(lib), "-lm"])
    return ctypes.CDLL(str(lib)).images


@pytest.mark.parametrize("L", [1.0, 1.999999, 15.5, 24.857860, 64.0, 99.43144, 1000.0, 1e4, 3e-3])
def test_equals_the_references_expression(images, L):
    rng = np.random.default_rng(3)
    edges = np.array([0.0, 0.5, 1.0, 1.5, 2.5, 0.5 * (1 - 2.0 ** -8), 0.5 * (1 + 2.0 ** -8), 1.4375, 1.2969])
    near = (edges[:, None] * L * (1 + np.arange(-40, 41) * 2.0 ** -53)).ravel()
    wide = (edges[:, None] * L * (1 + np.arange(-40, 41) * 2.0 ** -22)).ravel()
    d = np.concatenate([rng.uniform(-3 * L, 3 * L, 200_000), near, -near, wide, -wide, [1e300, np.inf, -np.inf, np.nan]])
    d = np.ascontiguousarray(d)
    a, b = np.empty_like(d), np.empty_like(d)
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    images(ctypes.c_long(len(d)), p(d), ctypes.c_double(L), p(a), p(b))
    assert np.array_equal(a, b, equal_nan=True)
