"""gm_div_rcp and gm_abs_ge (csrc/gm_exact_math.h), compiled as C11 without
contraction: the quotient's bits against the division (ordinary and special
significands, zero, tiny and huge numerators), the comparison against fabs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = """
#include "gm_exact_math.h"
long wrong(long n, const double *num, const double *den) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        if (!gm_ordinary(den[i])) continue;
        const double q = gm_div_rcp(num[i], den[i], 1.0 / den[i]), r = num[i] / den[i];
        bad += !(q == r || (q != q && r != r));
    }
    return bad;
}
long wrong_ge(long n, const double *v, const double *t) {
    long bad = 0;
    for (long i = 0; i < n; i++) bad += gm_abs_ge(v[i], t[i]) != (fabs(v[i]) >= t[i]);
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("exact_division")
    src, out = tmp / "m.c", tmp / "m.so"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(HERE), "geodesic-m_gb300", "csrc")
    subprocess.check_call(["gcc", "-std=c11", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc, str(src), "-o",
                           str(out), "-lm"])
    L = ctypes.CDLL(str(out))
    L.wrong.restype = L.wrong_ge.restype = ctypes.c_long
    return L


def call(f, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    return f(ctypes.c_long(len(a)), a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p))


def special(r, n, lo, hi):
    """Significands near 1, 2 and powers of two, exponents in [lo, hi]."""
    m = np.where(r.random(n) < 0.5, 1.0 + r.integers(0, 8, n) * 2.0 ** -52, 2.0 - r.integers(1, 9, n) * 2.0 ** -52)
    return m * 2.0 ** r.integers(lo, hi, n) * np.where(r.random(n) < 0.5, 1, -1)


def test_quotients_are_the_divisions(lib):
    r = np.random.default_rng(2)
    n = 4_000_000
    wide = lambda lo, hi: (1 + r.random(n)) * 2.0 ** r.uniform(lo, hi, n).astype(int) * np.where(r.random(n) < 0.5, 1, -1)  # noqa: E731
    assert call(lib.wrong, wide(-40, 10), wide(-12, 12)) == 0
    assert call(lib.wrong, wide(-1070, 1020), wide(-220, 220)) == 0
    assert call(lib.wrong, special(r, n, -60, 60), special(r, n, -60, 60)) == 0
    assert call(lib.wrong, special(r, n, -60, 60), wide(-20, 20)) == 0
    edge = np.array([0.0, -0.0, 5e-324, 1e-310, np.inf, -np.inf, np.nan, 2.0 ** 700, 2.0 ** -700, 1.7e308])
    assert call(lib.wrong, np.repeat(edge, 1000), wide(-20, 20)[:len(edge) * 1000]) == 0


def test_comparison_is_fabs(lib):
    r = np.random.default_rng(4)
    t = 10.0 ** r.uniform(-14, 2, 1_000_000)
    v = t * np.where(r.random(len(t)) < 0.5, 1, -1) * (1 + r.integers(-3, 4, len(t)) * 2.0 ** -52)
    v[:6] = [0.0, -0.0, np.nan, -np.nan, np.inf, -np.inf]
    assert call(lib.wrong_ge, v, t) == 0
