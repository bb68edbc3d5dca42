"""The fixed-point sin, cos and atan2 (fd_trig_fx.h) against the double-double ones (fd_trig.h), bit for bit wherever
they answer: random arguments, table points and the middles between them, quadrant and octant borders, extremes."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtomoc_gb300", "csrc")
SRC = r"""
#include "fd_trig.h"
#include "fd_trig_fx.h"
static int same(double a, double b) { return fdx_bits(a) == fdx_bits(b); }
/* out: [0] differing, [1] refused */
void sincos_check(long n, const double *x, long *out)
{
    for (long i = 0; i < n; i++) {
        double s, c;
        if (!fdx_sincos(x[i], &s, &c)) out[1]++;
        else out[0] += !same(s, fdt_sin(x[i])) || !same(c, fdt_cos(x[i]));
    }
}
void atan2_check(long n, const double *y, const double *x, long *out)
{
    for (long i = 0; i < n; i++) {
        double a;
        if (!fdx_atan2(y[i], x[i], &a)) out[1]++;
        else out[0] += !same(a, fdt_atan2(y[i], x[i]));
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    (d / "t.c").write_text(SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC, str(d / "t.c"), "-o",
                    str(d / "t.so"), "-lm"], check=True)
    return C.CDLL(str(d / "t.so"))


def ptr(a):
    return np.ascontiguousarray(a, dtype=np.float64).ctypes.data_as(C.POINTER(C.c_double))


def check(fn, *args):
    args = [np.ascontiguousarray(a, dtype=np.float64) for a in args]
    out = (C.c_long * 2)()
    fn(C.c_long(len(args[0])), *[ptr(a) for a in args], out)
    return out[0], out[1]


def around(v):
    return np.concatenate([v, np.nextafter(v, 99), np.nextafter(v, -99), v + 1e-9, v - 1e-9])


def test_sincos_equals_double_double(lib):
    rng = np.random.default_rng(1)
    for span in (16.0, 3.2, 0.02):
        bad, refused = check(lib.sincos_check, rng.uniform(-span, span, 300_000))
        assert bad == 0 and refused < 100
    j = np.arange(-650, 651)
    bad, _ = check(lib.sincos_check, np.concatenate([around(j * (np.pi / 128)), around((j + 0.5) * (np.pi / 128))]))
    assert bad == 0
    bad, refused = check(lib.sincos_check, [0.0, -0.0, 1e-300, 2.0**-31, 16.0, -1e6, np.inf, -np.inf, np.nan])
    assert bad == 0 and refused == 9   # left to the double-double functions


def test_atan2_equals_double_double(lib):
    rng = np.random.default_rng(2)
    for scale in (1.0, 1e-3, 1e-5):
        y, x = rng.uniform(-6400, 6400, (2, 300_000))
        bad, refused = check(lib.atan2_check, y * scale, x)
        assert bad == 0 and refused < 3000
        bad, refused = check(lib.atan2_check, y, x * scale)
        assert bad == 0 and refused < 3000
    th = np.concatenate([np.arange(256) * (np.pi / 128), (np.arange(256) + 0.5) * (np.pi / 128)])
    for r in (1.0, 1.4, 1.99999, 6371.0, 1e-9, 1e200):
        for eps in (0.0, 1e-15, -1e-15, 1e-8):
            bad, _ = check(lib.atan2_check, r * np.sin(th + eps), r * np.cos(th + eps))
            assert bad == 0
    v = rng.uniform(1, 2, 1000)
    for sy in (1, -1):
        for sx in (1, -1):
            bad, refused = check(lib.atan2_check, sy * v, sx * v)
            assert bad == 0 and refused == 0
    e = np.array([0.0, -0.0, 1.0, -1.0, 5e-324, 1e-308, np.inf, -np.inf, np.nan])
    y, x = [m.ravel() for m in np.meshgrid(e, e)]
    bad, refused = check(lib.atan2_check, y, x)
    assert bad == 0 and refused == len(y) - 4   # only |y| = |x| = 1 is answered
