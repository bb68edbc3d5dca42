"""The c2f kernel's walk up z against the oracle, bit for bit: part and block remainders, cells of one plane and
cells longer than a walked part, sizes that walk 1, 3, 6, 12 and 24 planes, more parts than
a grid has rows.  The slowness kernel's wide and plain forms against IEEE division: every
alignment of its arrays, lengths about a vector and a block.  The reciprocal against the division, for all floats."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fdtomoc_gb300 import build as B
from oracle_util import oracle_c2f

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,ig", [((2, 2, 2), (1, 1, 1)), ((3, 2, 25), (1, 1, 1)), ((2, 5, 2), (130, 1, 23)),
                                   ((9, 9, 3), (7, 3, 24)), ((4, 3, 4), (43, 1, 31)), ((6, 5, 9), (5, 9, 3)),
                                   ((41, 41, 4), (5, 5, 10)), ((41, 41, 7), (5, 5, 10)), ((41, 41, 13), (5, 5, 10)),
                                   ((41, 41, 20), (5, 5, 10)), ((2, 2, 2), (1, 1, 1_600_000))])
def test_c2f_walk_equals_oracle(gpu_lib, nc, ig):
    rng = np.random.default_rng(5)
    nxc, nyc, nzc = nc
    p = dict(nxc=nxc, nyc=nyc, nzc=nzc, h=0.3, igridx=[ig[0]] * (nxc - 1), igridy=[ig[1]] * (nyc - 1),
             igridz=[ig[2]] * (nzc - 1), x0=-7.3, y0=11.1, z0=-2.7)
    coarse = (2.0 + 6.0 * rng.random((2, nzc, nyc, nxc))).astype(np.float32)
    with gpu_lib.Context(0) as ctx:
        fine = gpu_lib.c2f(ctx, nxc, nyc, nzc, p["igridx"], p["igridy"], p["igridz"], p["x0"], p["y0"], p["z0"], p["h"], coarse)
    assert np.array_equal(fine.view(np.uint32), oracle_c2f(p, coarse).view(np.uint32))


@pytest.mark.parametrize("vo,so", [(0, 0), (1, 0), (0, 2), (3, 3), (2, 1)])
@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4096, 4099, 65539])
def test_slowness_forms(gpu_lib, vo, so, n):
    import torch
    v = np.random.default_rng(n).uniform(0.1, 9.0, n).astype(np.float32)
    v[:: 17] *= np.float32(1e-38)   # subnormal velocities, infinite and huge slownesses
    v[n // 2] = np.float32(np.inf)
    src = torch.zeros(n + 4, dtype=torch.float32, device="cuda")
    src[vo:vo + n] = torch.from_numpy(v).cuda()
    dst = torch.full((n + 8,), -1.0, dtype=torch.float32, device="cuda")
    with gpu_lib.Context(0) as ctx:
        ctx.velocity_to_slowness(src.data_ptr() + 4 * vo, dst.data_ptr() + 4 * so, n)
        torch.cuda.synchronize()
    got = dst.cpu().numpy()
    with np.errstate(over="ignore", divide="ignore"):
        want = np.float32(1.0) / v
    assert np.array_equal(got[so:so + n].view(np.uint32), want.view(np.uint32))
    assert (got[:so] == -1).all() and (got[so + n:] == -1).all()


def test_reciprocal_is_the_division(gpu_lib, tmp_path):
    out = str(tmp_path / "librecip.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "recip_check.cu")
    r = subprocess.run([B._nvcc()] + B.ARCH + B.NVFLAGS + ["-I" + B.CSRC, "-shared", "-cudart", "static", src, "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    counts = (C.c_ulonglong * 2)()
    assert C.CDLL(out).recip_check(counts) == 0
    assert counts[1] == 1 << 30 and counts[0] == 0
