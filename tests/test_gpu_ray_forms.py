"""The rays' derivative lists against the oracle, bit for bit: blocks that are not full, limits that end a ray or fill
its list, coarse cells as small as fine ones (several nodes entered at a time, and left and met again), coarse
coordinates out of order, repeated or ending inside the model."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))

import ray_cases as RC  # noqa: E402
from oracle_util import ray_lib  # noqa: E402

from fdtomoc_gb300 import rayderv as R  # noqa: E402

pytestmark = pytest.mark.gpu


def coarse(g, kind):
    """the case's grid with other coarse coordinates; the arrays to keep"""
    axes = [np.ctypeslib.as_array(p, shape=(n,)).copy() for p, n in ((g.gx, g.nxc), (g.gy, g.nyc), (g.gz, g.nzc))]
    if kind == "fine":
        axes = [np.linspace(a[0], a[-1], n).astype(np.float32) for a, n in zip(axes, (g.nx, g.ny, g.nz))]
    elif kind == "two":
        axes = [a[[0, -1]] for a in axes]
    elif kind == "long":
        axes = [np.linspace(axes[0][0], axes[0][-1], 8000).astype(np.float32)] + [a[[0, -1]] for a in axes[1:]]
    elif kind == "short":
        axes = [a[:-1] if len(a) > 2 else a for a in axes]
    elif kind == "unordered":
        axes = [np.concatenate([a[:1], a[:0:-1], a[-1:]]) for a in axes]
    elif kind == "repeated":
        axes = [np.concatenate([a, a[-1:]]) for a in axes]
    axes = [np.ascontiguousarray(a) for a in axes]
    out = R.RayGrid.from_buffer_copy(g)
    out.nxc, out.nyc, out.nzc = (len(a) for a in axes)
    out.gx, out.gy, out.gz = (a.ctypes.data_as(C.POINTER(C.c_float)) for a in axes)
    return out, axes


@pytest.mark.parametrize("kind,nobs,max_seg,cap", [
    ("spec", 1, 0, 0), ("spec", 3, 0, 0), ("spec", 31, 0, 0), ("spec", 33, 0, 0), ("spec", 95, 7, 0), ("spec", 96, 8, 0),
    ("spec", 64, 9, 0), ("spec", 50, 0, 8), ("spec", 50, 0, 37), ("fine", 130, 0, 0), ("fine", 70, 0, 100), ("two", 40, 0, 0),
    ("long", 35, 0, 0),
    ("short", 60, 0, 0), ("unordered", 60, 0, 0), ("repeated", 60, 0, 0)])
def test_ray_lists_equal_oracle(gpu_lib, tmp_path, kind, nobs, max_seg, cap):
    import torch
    sp = R.read_spec(RC.write_inputs(RC.make_case(2), str(tmp_path)))
    g, keep = R.grid_from_spec(sp)
    src, n0, _, fields = R.build_observations(sp, g, R.read_stations(sp["stafile"]), R.read_events(sp["locdfil"]))
    fields = [np.ascontiguousarray(f, dtype=np.float32) for f in R.load_fields(sp, g, fields)]
    g, keep = coarse(g, kind)
    rng = np.random.default_rng(nobs)
    obs = (R.RayObs * nobs)()
    for o in range(nobs):
        C.memmove(C.byref(obs[o]), C.byref(src[o % n0]), C.sizeof(R.RayObs))
        obs[o].ez = float(np.clip(obs[o].ez + rng.uniform(-1.0, 1.0), g.z0 + 0.1, g.z0 + (g.nz - 2) * g.h))
    ms, cp = max_seg or R.default_max_seg(g), cap or R.default_cap(g)
    want, idx, du = (R.RayResult * nobs)(), np.zeros(nobs * cp, np.int32), np.zeros(nobs * cp, np.float32)
    fp = (C.POINTER(C.c_float) * len(fields))(*[f.ctypes.data_as(C.POINTER(C.c_float)) for f in fields])
    assert ray_lib().fdr_trace(C.byref(g), fp, nobs, obs, 1, ms, cp, want, idx.ctypes.data_as(C.POINTER(C.c_int)),
                               du.ctypes.data_as(C.POINTER(C.c_float))) == 0
    dev = [torch.from_numpy(f).cuda() for f in fields]
    with gpu_lib.Context(0) as ctx:
        res, off, gi, gd = gpu_lib.raytrace(ctx, g, [t.data_ptr() for t in dev], obs, nobs, cap=cp, max_seg=ms)
    for o in range(nobs):
        w = want[o]
        assert (res[o].status, res[o].nseg) == (w.status, w.nseg), f"observation {o}"
        if w.status == R.RAY_OK:
            assert res[o].nnz == w.nnz and np.array_equal(gi[off[o]:off[o + 1]], idx[o * cp:o * cp + w.nnz]), f"observation {o}"
            assert np.array_equal(gd[off[o]:off[o + 1]].view(np.int32), du[o * cp:o * cp + w.nnz].view(np.int32))
        else:
            assert off[o] == off[o + 1]
