"""Location at the sizes where its kernels change form: fields on and off a 16-byte boundary, plane sizes that are
no multiple of four nodes, windows of one to a hundred divisions (float pairs up to 64, double beyond), S times
scaled from P fields, times of an event at a station (residuals near zero, where a float residual is least
certain).  Every result against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle_util import loc_grid, oracle_locate
from test_gpu_locate import gpu_grid, random_case, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,shape,ivs,kmin,div,off,shift", [
    (21, (2, 2, 2), 1, 0, (1, 1), 0, 3.0), (22, (5, 3, 7), 0, 1, (1, 2), 1, 3.0), (23, (9, 14, 6), 1, 2, (2, 64), 2, 0.0),
    (24, (12, 12, 9), 0, 0, (64, 3), 3, 0.0), (25, (17, 13, 11), 1, 11, (20, 20), 0, 3.0), (26, (11, 10, 8), 1, 2, (65, 4), 0, 0.0),
    (27, (31, 33, 12), 0, 2, (20, 20), 1, 1e-3)])
def test_gpu_location_forms(gpu_lib, seed, shape, ivs, kmin, div, off, shift):
    import torch
    lib = gpu_lib
    p, fl, keys, events = random_case(seed, *shape, ivs, 45)
    p["kmin"], (p["ndiv"], p["ndiv2"]) = kmin, div
    # origin time: the case's picks carry 3 s; shift says how much of it is left
    events = [[(f, float(np.float32(t - 3.0 + shift)), w, ph, gd) for f, t, w, ph, gd in ev] for ev in events if ev]
    grid_o = loc_grid(p)
    g = gpu_grid(lib, p)
    grid_o.ivs = g.ivs = ivs
    dev = []
    for k in keys:   # `off` floats past an aligned address
        buf = torch.zeros(fl[k].size + 4, dtype=torch.float32, device="cuda")
        buf[off:off + fl[k].size] = torch.from_numpy(np.ascontiguousarray(fl[k]).reshape(-1))
        dev.append(buf)
    with lib.Context(0) as ctx:
        got = lib.locate(ctx, g, [t.data_ptr() + 4 * off for t in dev], events)
    host = [np.ascontiguousarray(fl[k]) for k in keys]
    for e, ob in enumerate(events):
        want = oracle_locate(grid_o, host, ob)
        assert same(got[e], want) is None, (e, same(got[e], want))
