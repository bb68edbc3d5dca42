"""The stencils as four lanes of the solver evaluate them against the one-lane forms, which the bound on 2-D values is
tested against: the same bits, over the geometry of configs 1 and 2."""
import ctypes as C
import os
import subprocess
import tempfile

import pytest

from fdtomoc_gb300 import build as B
from fdtomoc_gb300 import formats
from fdtomoc_gb300 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [1, 2])
def test_four_lane_stencils_equal_one_lane_forms(gpu_lib, cfg, tmp_path):
    out = os.path.join(tempfile.mkdtemp(prefix="fdquad_"), "libquad.so")
    r = subprocess.run([B._nvcc()] + B.ARCH + B.NVFLAGS + ["-I" + B.CSRC, "-shared", "-cudart", "static",
                                                           os.path.join(HERE, "quad_check.cu"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    g, v, sts = W.config(cfg)
    par = tmp_path / "s.par"
    formats.write_par(par, W.par_for(g, sts[0], str(tmp_path / "vp.mod"), "s.ptimes"))
    st, _, _ = gpu_lib.station_from_par("par=" + str(par))
    counts = (C.c_ulonglong * 9)()
    fn = C.CDLL(out).quad_check
    fn.argtypes = [C.c_int] * 3 + [C.c_double] * 5 + [C.c_int, C.c_ulonglong, C.POINTER(C.c_ulonglong)]
    assert fn(st.nx, st.ny, st.nz, st.h, st.dq, st.df, st.z0r, st.y0, 1000, 777 + cfg, counts) == 0
    for kind in range(3):
        items, differ, rooted = counts[3 * kind:3 * kind + 3]
        assert items > 100_000 and rooted > 0.05 * items and rooted < items, (kind, items, rooted)
        assert differ == 0, (kind, items, differ)
