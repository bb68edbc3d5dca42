"""Location with divisions of few bits, where the places in a cell are short fractions and every tenth residual of a
refinement is a tie of two floats, listed and formed in double: windows of whole and partial tiles of phases, S times
scaled by a number of few bits, and picks that fit to the last place (nearly every residual listed, in several rounds a
tile).  Every result against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle_util import loc_grid, oracle_locate
from test_gpu_locate import gpu_grid, random_case, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,shape,ivs,div,vpvs,fit", [
    (41, (12, 11, 9), 1, (4, 4), 1.75, 0), (42, (10, 12, 8), 0, (8, 8), 1.75, 0), (43, (9, 9, 9), 0, (16, 2), 1.5, 0),
    (44, (13, 10, 7), 1, (32, 16), 1.75, 0), (45, (11, 12, 10), 0, (8, 16), 1.75, 1), (46, (8, 8, 8), 1, (16, 4), 1.75, 1)])
def test_gpu_location_ties(gpu_lib, seed, shape, ivs, div, vpvs, fit):
    import torch
    lib = gpu_lib
    p, fl, keys, events = random_case(seed, *shape, ivs, 45)
    p["ndiv"], p["ndiv2"] = div
    grid_o, g = loc_grid(p), gpu_grid(lib, p)
    grid_o.ivs = g.ivs = ivs
    grid_o.vpvs = g.vpvs = vpvs
    host = [np.ascontiguousarray(fl[k]) for k in keys]
    if fit:   # linear fields of short numbers and picks at a node: residuals and their differences of few bits
        z, y, x = np.indices(host[0].shape)
        host = [((k % 7 + 1) * x + (k % 5 + 1) * y + (k % 3 + 1) * z).astype(np.float32) / 64 + 1 for k in range(len(host))]
        n = tuple(s // 2 for s in host[0].shape)
        events = [[(f, float(host[f][n]) * (vpvs if ivs == 0 and ph == "S" else 1.0), w, ph, gd) for f, t, w, ph, gd in ev] for ev in events]
    events = [ev for ev in events if ev]
    dev = [torch.from_numpy(h.reshape(-1)).cuda() for h in host]
    with lib.Context(0) as ctx:
        got = lib.locate(ctx, g, [t.data_ptr() for t in dev], events)
    for e, ob in enumerate(events):
        want = oracle_locate(grid_o, host, ob)
        assert same(got[e], want) is None, (e, same(got[e], want))
