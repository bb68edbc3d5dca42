"""Grids whose solves take each form of a chunk's evaluation and release: a few nodes (thin and tiny grids),
many (wide faces), several faces at once (the forward sweep) and one (restarts from every wall, reached by a
slow layer between fast ones).  Time files against the oracle, byte for byte."""
import os

import numpy as np
import pytest

from fdtomoc_gb300 import workloads as W
from fdtomoc_gb300.formats import write_grid, write_par
from oracle_util import run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,axis", [(2, 2, 2, 0), (3, 2, 5, 1), (40, 3, 4, 0), (4, 44, 5, 1), (5, 4, 50, 2),
                                           (66, 64, 9, 2), (9, 65, 40, 0), (65, 9, 40, 1), (33, 32, 31, 2)])
def test_chunk_forms(gpu_lib, tmp_path, nx, ny, nz, axis):
    g = W.Grid(nx, ny, nz, 0.01, 0.01, 1.0)
    rng = np.random.default_rng(nx * 10000 + ny * 100 + nz)
    k = np.indices((nz, ny, nx))[2 - axis] / max(1, (nx, ny, nz)[axis] - 1)
    v = (np.where(k < 0.3, 6.0, np.where(k < 0.6, 3.5, 8.0)) * (1 + 0.03 * rng.standard_normal((nz, ny, nx)))).astype(np.float32)
    write_grid(str(tmp_path / "vp.mod"), W.head_for(g), v)
    entries = []
    for i, (fx, fy) in enumerate([(0.5, 0.5), (0.1, 0.85)]):
        st = dict(lon=g.x0 + fx * (nx - 1) * g.dlon, lat=g.y0 - fy * (ny - 1) * g.dlat, elev=1.5 - i)
        pf = str(tmp_path / f"s{i}.par")
        write_par(pf, W.par_for(g, st, str(tmp_path / "vp.mod"), f"s{i}.ptimes"))
        run_oracle(pf, str(tmp_path / "orc"))
        entries.append("par=" + pf)
    os.makedirs(tmp_path / "gpu", exist_ok=True)
    assert gpu_lib.sphfd_parlist(entries, str(tmp_path / "gpu")) == [0, 0]
    for i in range(2):
        a, b = (open(tmp_path / d / f"s{i}.ptimes", "rb").read() for d in ("orc", "gpu"))
        assert a == b
