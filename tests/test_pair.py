"""The location's residuals in pairs of floats (fd_pair.h), at nodes and between them, against the reference's double form: the pair within its
margin of it, and every residual called certain the same float.  P phases and S phases scaled from a P field, near-zero
residuals (where a float is least certain) among them, times up to 300 s that differ by 0.1 ms to 1 s within the
cell, places on steps of the usual divisions, and places beyond the cell along z."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtomoc_gb300", "csrc")
SRC = r"""
#include <stdint.h>
#include "fd_pair.h"
static uint64_t s;
static double uni(void)
{
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return (double)(s >> 11) * 0x1p-53;
}
/* src/sphfdloc.c's find_time and residual, term by term */
static double residual(float obs, int scaled, float vpvs, const float *t, double fx, double fy, double fz)
{
    const double w[8] = {(1.0 - fx) * (1.0 - fy) * (1.0 - fz), fx * (1.0 - fy) * (1.0 - fz), (1.0 - fx) * fy * (1.0 - fz),
                         (1.0 - fx) * (1.0 - fy) * fz, fx * fy * (1.0 - fz), fx * (1.0 - fy) * fz, (1.0 - fx) * fy * fz,
                         fx * fy * fz};
    const int at[8] = {0, 1, 2, 4, 3, 5, 6, 7};
    double tp = 0.;
    for (int i = 0; i < 8; i++) tp += w[i] * t[at[i]];
    return scaled ? (double)obs - tp * (double)vpvs : (double)obs - tp;
}
/* out: [0] pairs outside their margin, [1] certain but another float, [2] certain */
void pair_check(uint64_t seed, long n, int scaled, double vpvs_, int ndiv, int beyond, double near, long *out)
{
    const float vpvs = (float)vpvs_;
    s = seed;
    for (long i = 0; i < n; i++) {
        const double far = 0.3 * pow(1000., uni()), span = pow(10., -4. + 4. * uni());
        float t[8], m, res;
        for (int k = 0; k < 8; k++) t[k] = (float)(far + span * uni());
        double f[3];
        for (int k = 0; k < 3; k++) f[k] = ndiv ? floor(uni() * (ndiv + 1)) / ndiv : uni();
        if (beyond) f[2] += 1.;
        const float obs = (float)(-residual(0.f, scaled, vpvs, t, f[0], f[1], f[2]) + near * (uni() - .5));
        const float fh = (float)f[0], fl = (float)(f[0] - fh);
        fdp_ff w[4];
        fdp_row ab;
        fdp_weights(fdp_pair((float)f[1], (float)(f[1] - (float)f[1])), fdp_pair((float)f[2], (float)(f[2] - (float)f[2])), w);
        fdp_coefficients(obs, scaled, vpvs, t, 2, 4, w, &ab, &m);
        const double want = residual(obs, scaled, vpvs, t, f[0], f[1], f[2]);
        const double have = (double)ab.ah + (double)ab.al - ((double)ab.bh + (double)ab.bl) * f[0];
        out[0] += !(fabs(have - want) <= m);
        if (fdp_residual(&ab, m, fh, fl, &res)) {
            out[2]++;
            out[1] += res != (float)want;
        }
    }
}
/* out: [0] certain but another float, [1] certain */
void node_check(uint64_t seed, long n, double vpvs_, int mode, long *out)
{
    const float vpvs = (float)vpvs_;
    s = seed;
    for (long i = 0; i < n; i++) {
        float t = (float)(0.3 * pow(1000., uni())), obs, res;
        if (mode == 0) obs = (float)((double)t * vpvs + 4. * (uni() - .5));          /* a pick's residual */
        else if (mode == 1) obs = (float)((double)t * vpvs);                         /* none but a rounding */
        else if (mode == 2) obs = (float)(t * pow(2., 60. * uni() - 30.) * (uni() < .5 ? -1. : 1.));   /* far apart */
        else {   /* few bits: ties at every size */
            t = (float)ldexp((double)(1 + (int)(uni() * 0xffffff)), (int)(uni() * 40.) - 20);
            obs = (float)ldexp((double)(1 + (int)(uni() * 255.)), (int)(uni() * 60.) - 30);
        }
        if (fdp_scaled_residual(obs, t, vpvs, &res)) {
            out[1]++;
            out[0] += res != (float)((double)obs - (double)t * (double)vpvs);
        }
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair")
    (d / "t.c").write_text(SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC, str(d / "t.c"), "-o",
                    str(d / "t.so"), "-lm"], check=True)
    return C.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("scaled,vpvs", [(0, 1.0), (1, 1.78), (1, 1.732), (1, 0.5), (1, -1.7)])
@pytest.mark.parametrize("ndiv,beyond", [(0, 0), (20, 0), (8, 0), (0, 1)])
def test_pair_residual_within_its_margin(lib, scaled, vpvs, ndiv, beyond):
    out = (C.c_long * 3)()
    for k, near in enumerate((0.0, 1e-3, 1.0)):
        lib.pair_check(C.c_uint64(88172645463325252 + k), C.c_long(150_000), scaled, C.c_double(vpvs), ndiv, beyond,
                       C.c_double(near), out)
    assert out[0] == 0, f"{out[0]} pairs outside their margin"
    assert out[1] == 0, f"{out[1]} certain residuals that are another float"
    assert out[2] > 100_000   # most are certain away from zero


@pytest.mark.parametrize("vpvs", [1.75, 1.5, 2.0, 1.78, 1.0, -1.75, 1.7320508])
def test_scaled_node_residual(lib, vpvs):
    """Certain residuals are the reference's float; ties, of which a factor of few bits makes many, are certain too."""
    for mode in range(4):
        out = (C.c_long * 2)()
        lib.node_check(C.c_uint64(88172645463325252 + mode), C.c_long(400_000), C.c_double(vpvs), mode, out)
        assert out[0] == 0, f"{out[0]} certain residuals that are another float"
        if mode < 2:
            assert out[1] > 0.999 * 400_000, out[1]
