"""gm_rsqrt_step (csrc/gm_exact_math.h), compiled as C11 without contraction:
within 1.002 ulp of 1 / sqrt(x) for every seed as far off as the GPU's own can
be.  The bound: half an ulp for the result's rounding, half for the rounding of
x y (2^-54 relative), 2^-11 ulp for the series' next term.  The seed is FP32, of
x truncated to FP32 (2^-24 of the root), with the approximate instruction's
documented error of 2^-22.9."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = """
#include "gm_exact_math.h"
double worst(long n, const double *x, const double *off) {
    double w = 0.0;
    for (long i = 0; i < n; i++) {
        const long double r = 1.0L / sqrtl((long double)x[i]);
        const double y = (double)(float)((double)r * (1.0 + off[i]));
        const double v = gm_rsqrt_step(x[i], y);
        const double near = (double)r, ulp = nextafter(near, 1e300) - near;
        const double err = fabs((double)(((long double)v - r) / (long double)ulp));
        if (!(err <= w)) w = err;
    }
    return w;
}
"""


@pytest.fixture(scope="module")
def worst(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("reciprocal_root")
    src, lib = tmp / "m.c", tmp / "m.so"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(HERE), "geodesic-m_gb300", "csrc")
    subprocess.check_call(["gcc", "-std=c11", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc, str(src), "-o",
                           str(lib), "-lm"])
    f = ctypes.CDLL(str(lib)).worst
    f.restype = ctypes.c_double

    def call(x, off):
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        return f(ctypes.c_long(len(x)), p(x), p(off))
    return call


@pytest.mark.parametrize("lo,hi", [(-4, 10), (-100, 100)])
def test_within_an_ulp(worst, lo, hi):
    r = np.random.default_rng(6)
    n = 2_000_000
    x = np.ascontiguousarray((1 + r.random(n)) * 2.0 ** r.integers(lo, hi, n))
    x[:1000] = 2.0 ** r.integers(lo, hi, 1000) * (1 + r.integers(0, 4, 1000) * 2.0 ** -52)
    # the seed's error, the truncation's included; the rounding to FP32 above adds its own
    far = 2.0 ** -22.9 + 2.0 ** -24
    off = np.where(r.random(n) < 0.5, r.uniform(-far, far, n), np.where(r.random(n) < 0.5, far, -far))
    assert worst(x, np.ascontiguousarray(off)) <= 1.002
