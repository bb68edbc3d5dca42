"""Windows with a fast layer at an edge of the grid, where many border points need the stencil state of an earlier
point before their instance's order is known (a bound on the missing times stands in for it): time files
against the oracle, byte for byte.  The last grid's faces are too large for the bound's flags, the one before has
more open nodes than it looks through."""
import os

import numpy as np
import pytest

from fdtomoc_gb300 import workloads as W
from fdtomoc_gb300.formats import write_grid, write_par
from oracle_util import run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,axis,flip", [(31, 29, 23, 2, 0), (33, 32, 11, 2, 0), (25, 47, 30, 0, 1), (40, 33, 29, 1, 0),
                                                (24, 24, 44, 2, 1), (160, 150, 12, 2, 0), (215, 213, 4, 2, 0)])
def test_deferred_points(gpu_lib, tmp_path, nx, ny, nz, axis, flip):
    g = W.Grid(nx, ny, nz, 0.01, 0.01, 1.0)
    rng = np.random.default_rng(nx * 10000 + ny * 100 + nz)
    k = np.indices((nz, ny, nx))[2 - axis] / max(1, (nx, ny, nz)[axis] - 1)
    k = 1 - k if flip else k
    v = ((3.0 + 5.0 * k ** 3) * (1 + 0.05 * rng.standard_normal((nz, ny, nx)))).astype(np.float32)
    write_grid(str(tmp_path / "vp.mod"), W.head_for(g), v)
    entries = []
    for i, (fx, fy, fz) in enumerate([(0.5, 0.5, 0.3), (0.15, 0.8, 0.6)]):
        st = dict(lon=g.x0 + fx * (nx - 1) * g.dlon, lat=g.y0 - fy * (ny - 1) * g.dlat, elev=1.5 - i)
        pf = str(tmp_path / f"s{i}.par")
        write_par(pf, W.par_for(g, st, str(tmp_path / "vp.mod"), f"s{i}.ptimes"))
        run_oracle(pf, str(tmp_path / "orc"))
        entries.append("par=" + pf)
    os.makedirs(tmp_path / "gpu", exist_ok=True)
    assert gpu_lib.sphfd_parlist(entries, str(tmp_path / "gpu")) == [0, 0]
    deferred = 0
    for i, e in enumerate(entries):
        a, b = (open(tmp_path / d / f"s{i}.ptimes", "rb").read() for d in ("orc", "gpu"))
        assert a == b
        st, _, _ = gpu_lib.station_from_par(e)
        with gpu_lib.Context(0) as ctx:
            _, (stats,) = ctx.solve_host([st], v)
        deferred += stats["deferred"]
    assert deferred > 0
