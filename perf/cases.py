"""Cases that stand for what a program does with this framework, each through a public entry point.

One iteration of a tomographic inversion interpolates the coarse model onto the fine grid (c2f), turns
velocities into slowness, solves travel-time fields for its stations (alone, as one batch, from host
arrays, or through a serving session), locates the events in those fields and traces the rays back
through them.  The solves carry the path: a station field takes from milliseconds (a 27x20x21 test
grid) to about ten seconds (a 301x301x121 window of the benchmark).  The cases here keep a pass below
two seconds, so the largest of them fills the GPU with windows of about 80 nodes a side, whose arrays
together are far larger than the L2, and a lone station has up to about half a million nodes.

Models follow the benchmark's recipe (a layered profile times a smooth perturbation), travel-time
fields for the location and ray cases are closed-form times in a medium whose velocity grows linearly
with depth, scaled by a smooth factor so that rays bend.
"""
import ctypes
import math

import numpy as np
import torch

from fdtomoc_gb300 import lib
from fdtomoc_gb300 import rayderv as R
from fdtomoc_gb300 import workloads as W

# the catalog cases' fields stay on the GPU as the solver left them: one float32 grid per station


def listed():
    return [
        # a small regional test grid, solved on its own: launch and host work weigh the most
        dict(name="solve 27x20x21", op="solve", nx=27, ny=20, nz=21, step=0.01, n=1),
        # the plain one-station solve of the smallest benchmark grid
        dict(name="solve 61x61x31", op="solve", nx=61, ny=61, nz=31, step=0.01, n=1),
        # one ragged window of the uneven workload alone: a station asked for by itself
        dict(name="solve window 141x121x57", op="solve", nx=141, ny=121, nz=57, step=0.005, n=1),
        # uneven windows in one prepared batch, three waves of stations on the GPU
        dict(name="batch 400 windows 25..61", op="batch", n=400, lo=25, hi=61, hiz=41, mx=161, mz=81),
        # a full GPU of the larger windows: one station per SM, arrays far beyond the L2
        dict(name="batch 150 windows 73..91", op="batch", n=150, lo=73, hi=91, hiz=53, mx=301, mz=81),
        # host arrays in and out, as the drop-in program calls it: one station list, one velocity file
        dict(name="host 24 stations 49x45x33", op="host", nx=49, ny=45, nz=33, step=0.01, n=24),
        # P and S requests of mixed windows through a serving session
        dict(name="serve 48 requests 31..61", op="serve", n=48, lo=31, hi=61, hiz=41, mx=121, mz=61),
        # one event just picked, against the fields of a small network
        dict(name="locate 1 event 61x61x31", op="locate", nx=61, ny=61, nz=31, step=0.01, stations=12, events=1,
             scaled=False),
        # a catalog against the benchmark's 64 stations
        dict(name="locate 128 events 201x201x81", op="locate", nx=201, ny=201, nz=81, step=0.005, stations=64,
             events=128, scaled=False),
        # the rays of the benchmark's catalog, a quarter of its events
        dict(name="rays 256 events 201x201x81", op="rays", cx=10, cz=5, nxc=21, nzc=17, step=0.005, stations=64,
             events=256),
        # the fine P and S model of the largest workload from its coarse nodes, plan kept
        dict(name="c2f 401x401x161", op="c2f", nxc=41, nyc=41, nzc=33, cx=10, cz=5),
        # the fine model's slowness, once per model and iteration
        dict(name="slowness 401x401x161", op="slowness", nx=401, ny=401, nz=161),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    op = rng.choice(["solve", "solve", "batch", "batch", "host", "serve", "locate", "locate", "rays", "rays", "c2f",
                     "slowness"])
    if op == "solve":
        return dict(op=op, nx=log_int(13, 93), ny=log_int(13, 93), nz=log_int(9, 41), step=rng.choice([0.005, 0.01]),
                    n=log_int(1, 6))
    if op == "host":
        return dict(op=op, nx=log_int(13, 61), ny=log_int(13, 61), nz=log_int(9, 33), step=rng.choice([0.005, 0.01]),
                    n=log_int(2, 40))
    if op == "batch":
        lo = log_int(13, 61)
        return dict(op=op, n=log_int(8, 240), lo=lo, hi=lo + log_int(4, 24), hiz=rng.randint(21, 45), mx=121, mz=61)
    if op == "serve":
        lo = log_int(13, 45)
        return dict(op=op, n=log_int(4, 96), lo=lo, hi=lo + log_int(4, 20), hiz=rng.randint(17, 41), mx=101, mz=51)
    if op == "locate":
        return dict(op=op, nx=log_int(31, 201), ny=log_int(31, 201), nz=log_int(17, 81),
                    step=rng.choice([0.005, 0.01]), stations=rng.randint(9, 64), events=log_int(1, 120),
                    scaled=rng.random() < 0.3)
    if op == "rays":
        return dict(op=op, cx=rng.randint(3, 10), cz=rng.randint(2, 5), nxc=rng.randint(5, 21),
                    nzc=rng.randint(4, 17), step=rng.choice([0.005, 0.01]), stations=rng.randint(6, 64),
                    events=log_int(1, 256))
    if op == "c2f":
        return dict(op=op, nxc=log_int(3, 41), nyc=log_int(3, 41), nzc=log_int(3, 33), cx=rng.randint(2, 10),
                    cz=rng.randint(1, 5))
    return dict(op=op, nx=log_int(27, 401), ny=log_int(20, 401), nz=log_int(21, 161))


# ---- inputs ------------------------------------------------------------------------------------


def _noise(shape, spacing_km, corr_km, seed):
    """Gaussian-smoothed noise with largest value 1, as workloads.smooth_noise, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda"))
    k = [torch.fft.fftfreq(n, d, device="cuda") for n, d in zip(shape[:2], spacing_km[:2])]
    k.append(torch.fft.rfftfreq(shape[2], spacing_km[2], device="cuda"))
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    g = torch.fft.irfftn(r * torch.exp(-2.0 * (math.pi * corr_km) ** 2 * k2), s=shape)
    return g / g.abs().max()


def _grid(nx, ny, nz, step):
    return W.Grid(nx, ny, nz, step, step, 100.0 * step)


def _model(g, seed):
    """The benchmark's layered profile with a 5 % (0.01-degree grids: 3 %) smooth perturbation."""
    fine = g.dlat < 0.008
    v1 = torch.from_numpy(W.vp_1d(g.z0 + g.h * np.arange(g.nz)).astype(np.float32)).cuda()
    km = (g.h, g.dlat * W.KM_PER_DEG, g.dlon * W.KM_PER_DEG * math.cos(math.radians(g.y0)))
    return (v1[:, None, None] * (1.0 + (0.05 if fine else 0.03) * _noise(g.shape, km, 10.0 if fine else 5.0, seed)))


def _station(par):
    return lib.station_from_par(*[f"{k}={v}" for k, v in par.items()])[0]


def _stations(g, n, seed):
    return [_station(W.par_for(g, s, "vp.mod", "t")) for s in W.stations(g, n, seed)]


def _windows(g, n, lo, hi, hiz, seed):
    """Uneven windows of the model, each with a surface station inside it.  The sizes are the case's; where
    the windows and the stations lie comes from the seed."""
    size, rng = np.random.default_rng(n * 1000 + hi), np.random.default_rng(seed)
    out = []
    for _ in range(n):
        wx, wy = int(size.integers(lo, hi + 1)), int(size.integers(lo, hi + 1))
        wz = int(size.integers(min(lo, 21), hiz + 1))
        ox, oy = int(rng.integers(0, g.nx - wx + 1)), int(rng.integers(0, g.ny - wy + 1))
        w = dict(nx=wx, ny=wy, nz=wz, ox=ox, oy=oy, fx=float(rng.uniform(2, wx - 3)),
                 fy=float(rng.uniform(2, wy - 3)), elev=float(rng.uniform(0, 2)))
        st = _station(W.window_par(g, w, "vp.mod", "t"))
        st.ox, st.oy, st.oz = ox, oy, 0
        out.append(st)
    return out


def _fields(sts):
    """One device buffer for all fields, each on a 256-byte boundary, and the fields' addresses."""
    at, off = 0, []
    for s in sts:
        off.append(at)
        at += (s.nx * s.ny * s.nz + 63) // 64 * 64
    flat = torch.zeros(at, dtype=torch.float32, device="cuda")
    return flat, [flat.data_ptr() + 4 * o for o in off], off


_SHARED = {}


def _stream():
    """The program's stream."""
    if "stream" not in _SHARED:
        _SHARED["stream"] = torch.cuda.Stream()
    return _SHARED["stream"].cuda_stream


def _slowness(ctx, v):
    s = torch.empty_like(v)
    torch.cuda.synchronize()
    ctx.velocity_to_slowness(v.data_ptr(), s.data_ptr(), v.numel(), _stream())
    torch.cuda.synchronize()
    return s


def _network(case, seed):
    """Location / ray grid of the fields, stations in its frame (radians, km), and one closed-form field
    per station."""
    rng = np.random.default_rng(seed)
    if case["op"] == "rays":
        nx = ny = 1 + case["cx"] * (case["nxc"] - 1)
        nz = 1 + case["cz"] * (case["nzc"] - 1)
        step = case["step"]
        sp = dict(nxc=case["nxc"], nyc=case["nxc"], nzc=case["nzc"], igridx=[case["cx"]] * (case["nxc"] - 1),
                  igridy=[case["cx"]] * (case["nxc"] - 1), igridz=[case["cz"]] * (case["nzc"] - 1), h=100.0 * step,
                  x0=120.5, y0=23.5, z0=-2.0, dq=step, df=step)
        g, keep = R.grid_from_spec(sp, spacing_rule=False)
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        g, keep = lib.loc_grid_from_spec(nx, ny, nz, 120.5, 23.5, -2.0, 100.0 * case["step"]), None
    sts = [dict(xs=g.x0 + g.df * rng.uniform(2, nx - 3), ys=g.y0 + g.dq * rng.uniform(2, ny - 3),
                zs=-float(rng.uniform(0.0, 1.9)), kx=rng.uniform(1, 3), ky=rng.uniform(1, 3), amp=rng.uniform(0, 0.04))
           for _ in range(case["stations"])]
    lon = torch.from_numpy(g.x0 + g.df * np.arange(nx)).cuda()[None, None, :]
    col = torch.from_numpy(g.y0 + g.dq * np.arange(ny)).cuda()[None, :, None]
    dep = torch.from_numpy(g.z0 + g.h * np.arange(nz)).cuda()[:, None, None]
    fields = [_time(g, nx, ny, s, lon, col, dep, torch).to(torch.float32).contiguous() for s in sts]
    return g, keep, sts, fields, (nx, ny, nz), rng


def _time(g, nx, ny, s, lon, col, dep, m):
    """Time from station s: a linear velocity 5 + 0.06 z km/s between the end points' straight distance,
    times a smooth factor."""
    def xyz(a, b, z):
        r = 6371.0 - z
        return r * m.sin(b) * m.cos(a), r * m.sin(b) * m.sin(a), r * m.cos(b)
    x, y, z = xyz(lon, col, dep)
    one = torch.tensor if m is torch else np.float64
    kw = dict(dtype=torch.float64, device="cuda") if m is torch else {}
    sx, sy, sz = xyz(*(one(s[k], **kw) for k in ("xs", "ys", "zs")))
    d2 = (x - sx) ** 2 + (y - sy) ** 2 + (z - sz) ** 2
    a = 0.06
    v1, v2 = 5.0 + a * (dep + 2.0), 5.0 + a * (s["zs"] + 2.0)
    acosh = m.acosh if m is torch else np.arccosh
    t = acosh(1.0 + a * a * d2 / (2.0 * v1 * v2)) / a
    u, v = (lon - g.x0) / (g.df * (nx - 1)), (col - g.y0) / (g.dq * (ny - 1))
    return t * (1.0 + s["amp"] * m.sin(s["kx"] * math.pi * u) * m.cos(s["ky"] * math.pi * v))


def _picks(g, dims, sts, rng, count, floor):
    """One event inside the grid and the stations that recorded it: (hypocentre, station numbers).  How
    many did is the case's (count), which ones comes from the seed."""
    nx, ny, nz = dims
    h = (g.x0 + g.df * rng.uniform(3, nx - 4), g.y0 + g.dq * rng.uniform(3, ny - 4),
         g.z0 + g.h * rng.uniform(floor, nz - 4))
    most = min(len(sts), 40)
    return h, rng.choice(len(sts), size=int(count.integers(min(most, 24), most + 1)), replace=False)


def prepare(case, seed):
    op = case["op"]
    if op in ("solve", "host"):
        g = _grid(case["nx"], case["ny"], case["nz"], case["step"])
        st = dict(op=op, ctx=lib.Context(0), sts=_stations(g, case["n"], seed), v=_model(g, seed))
        if op == "host":
            st["v"] = st["v"].cpu().numpy()
            return st
        st["slow"] = _slowness(st["ctx"], st["v"])
        st["flat"], st["ptrs"], _ = _fields(st["sts"])
        st["dims"] = (g.nx, g.nx * g.ny)
        return st
    if op == "batch":
        g = _grid(case["mx"], case["mx"], case["mz"], 0.005)
        st = dict(op=op, ctx=lib.Context(0), sts=_windows(g, case["n"], case["lo"], case["hi"], case["hiz"], seed))
        st["slow"] = _slowness(st["ctx"], _model(g, seed))
        st["flat"], ptrs, _ = _fields(st["sts"])
        st["batch"] = lib.Batch(st["ctx"], st["sts"], st["slow"].data_ptr(), g.nx, g.nx * g.ny, ptrs)
        return st
    if op == "serve":
        g = _grid(case["mx"], case["mx"], case["mz"], 0.005)
        vp = _model(g, seed)
        vs = vp / 1.73 * (1.0 + 0.02 * _noise(g.shape, (0.5, 0.556, 0.509), 10.0, seed + 1))
        sts = _windows(g, case["n"], case["lo"], case["hi"], case["hiz"], seed)
        flat, _, off = _fields(sts)
        outs = [flat[o:o + s.nx * s.ny * s.nz] for s, o in zip(sts, off)]
        srv = lib.Server(0, hbm_bytes=6 << 30)
        srv.set_model(0, vp.contiguous())
        srv.set_model(1, vs.contiguous())
        return dict(op=op, srv=srv, sts=sts, outs=outs, flat=flat)
    if op == "locate":
        g, _, sts, fields, dims, rng = _network(case, seed)
        if case["scaled"]:
            g.ivs, g.vpvs = 0, 1.75     # one model: S times are the P field's times vpvs
        events, count = [], np.random.default_rng(case["events"])
        for _ in range(case["events"]):
            (ex, ey, ez), sel = _picks(g, dims, sts, rng, count, 3)
            ob, origin = [], rng.uniform(-1.0, 1.0)    # the catalog's origin time is about a second off
            for s in sel:
                ph = "S" if case["scaled"] and rng.random() < 0.4 else "P"
                t = float(_time(g, dims[0], dims[1], sts[s], ex, ey, ez, np)) * (1.75 if ph == "S" else 1.0)
                t += origin + rng.normal(0, 0.02) + (rng.choice([-1.5, 2.5]) if rng.random() < 0.05 else 0.0)
                w = np.float32(rng.choice([0.05, 0.1, 0.2]))
                ob.append((int(s), float(np.float32(t)), float(np.float32(1.0) / (w * w)), ph, 1))
            events.append(ob)
        return dict(op=op, ctx=lib.Context(0), grid=g, events=events, fields=fields,
                    ptrs=[f.data_ptr() for f in fields])
    if op == "rays":
        g, keep, sts, fields, dims, rng = _network(case, seed)
        obs, count = [], np.random.default_rng(case["events"])
        for _ in range(case["events"]):
            (ex, ey, ez), sel = _picks(g, dims, sts, rng, count, 5 if dims[2] > 12 else 2)
            for s in sel:
                w = np.float32(rng.choice([0.05, 0.1, 0.2]))
                obs.append(R.RayObs(ex, ey, ez, sts[s]["xs"], sts[s]["ys"], sts[s]["zs"], int(s), 0,
                                    float(np.float32(rng.uniform(5, 40))), float(np.float32(1.0) / (w * w)), 0.0, 0))
        return dict(op=op, ctx=lib.Context(0), grid=g, keep=keep, obs=(R.RayObs * len(obs))(*obs), n=len(obs),
                    fields=fields, ptrs=[f.data_ptr() for f in fields])
    ctx = lib.Context(0)
    if op == "c2f":
        rng = np.random.default_rng(seed)
        nxc, nyc, nzc = case["nxc"], case["nyc"], case["nzc"]
        vp = 5.0 + 0.1 * np.arange(nzc)[:, None, None] + 0.2 * rng.random((nzc, nyc, nxc))
        coarse = torch.from_numpy(np.stack([vp, vp / 1.73]).astype(np.float32)).cuda()
        spec = (nxc, nyc, nzc, [case["cx"]] * (nxc - 1), [case["cx"]] * (nyc - 1), [case["cz"]] * (nzc - 1),
                -100.0, -100.0, -2.0, 0.5)
        plan = lib.C2fPlan(ctx, *spec)
        return dict(op=op, ctx=ctx, plan=plan, coarse=coarse, spec=spec,
                    fine=torch.empty(plan.shape, dtype=torch.float32, device="cuda"))
    g = _grid(case["nx"], case["ny"], case["nz"], 0.005)
    v = _model(g, seed).contiguous()
    return dict(op=op, ctx=ctx, v=v, slow=torch.empty_like(v))


# ---- one pass ----------------------------------------------------------------------------------


def run(state):
    op = state["op"]
    if op == "solve":
        nx, nxy = state["dims"]
        stats = state["ctx"].solve_device(state["sts"], state["slow"].data_ptr(), nx, nxy, state["ptrs"],
                                          stream_ptr=_stream())
        return dict(times=state["flat"], sweeps=[s["sweeps"] for s in stats][:8],
                    updates=sum(s["node_updates"] for s in stats))
    if op == "host":
        times, stats = state["ctx"].solve_host(state["sts"], state["v"])
        return dict(times=times, updates=sum(s["node_updates"] for s in stats))
    if op == "batch":
        state["batch"].run(_stream())
        return dict(times=state["flat"])
    if op == "serve":
        srv, n = state["srv"], len(state["sts"])
        for k, (st, out) in enumerate(zip(state["sts"], state["outs"])):
            srv.submit(st, k % 2, out, tag=k)
        done = []
        while len(done) < n:
            done += srv.poll(n, 60000)
        return dict(times=state["flat"], status=sum(abs(r["status"]) for r in done))
    if op == "locate":
        out = lib.locate(state["ctx"], state["grid"], state["ptrs"], state["events"], _stream())
        got = {k: np.array([r[k] for r in out]) for k in ("exm", "eym", "ezm", "stdmin", "status", "ngood", "passes")}
        for k in ("resmin", "tps"):
            got[k] = np.array([x for r in out for x in r[k]], np.float32)
        got["good"] = np.array([x for r in out for x in r["good"]])
        return got
    if op == "rays":
        res, off, idx, du = lib.raytrace(state["ctx"], state["grid"], state["ptrs"], state["obs"], state["n"],
                                         stream_ptr=_stream(), total_cap=256 * state["n"])
        r = np.ctypeslib.as_array(res)[:state["n"]]
        # the packed derivatives with the room behind them: as many values for every seed
        return dict(dt=r["dt"], am=r["am"], status=r["status"], nseg=r["nseg"], off=off, idx=idx.base, du=du.base)
    if op == "c2f":
        state["plan"].run(state["coarse"].data_ptr(), state["fine"].data_ptr(), _stream())
        return state["fine"]
    state["ctx"].velocity_to_slowness(state["v"].data_ptr(), state["slow"].data_ptr(), state["v"].numel(), _stream())
    return state["slow"]


# ---- what a pass cannot do without -----------------------------------------------------------------

# FP64 operations of one node update: a corner stencil (116) and a few one-step trials
_UPDATE = 150


def work(case):
    op = case["op"]
    if op in ("solve", "host"):
        n = case["nx"] * case["ny"] * case["nz"]
        model = 2 if op == "host" else 1    # velocity in, then slowness, where the model comes from the host
        return dict(bytes=4 * n * (case["n"] + model), flops=_UPDATE * n * case["n"])
    if op in ("batch", "serve"):
        n = int(case["n"] * (0.5 * (case["lo"] + case["hi"])) ** 2 * 0.5 * (min(case["lo"], 21) + case["hiz"]))
        return dict(bytes=4 * (n + case["mx"] ** 2 * case["mz"]), flops=_UPDATE * n)
    picks = case["events"] * 0.5 * (min(case["stations"], 24) + min(case["stations"], 40)) if "events" in case else 0
    if op == "locate":
        n = case["nx"] * case["ny"] * (case["nz"] - 2)
        # five float operations per pick and node, about 20 per pick and point of the two refinements
        return dict(bytes=4 * n * case["stations"], flops=picks * (5 * n + 2 * 41 ** 3 * 20))
    if op == "rays":
        cells = 0.6 * (2 * case["cx"] * (case["nxc"] - 1) + case["cz"] * (case["nzc"] - 1)) / 1.5
        return dict(bytes=picks * (cells * 32 + 64), flops=picks * cells * 1500)
    if op == "c2f":
        n = (1 + case["cx"] * (case["nxc"] - 1)) * (1 + case["cx"] * (case["nyc"] - 1)) * (1 + case["cz"] * (case["nzc"] - 1))
        return dict(bytes=8 * (n + case["nxc"] * case["nyc"] * case["nzc"]), flops=2 * 31 * n)
    n = case["nx"] * case["ny"] * case["nz"]
    return dict(bytes=8 * n, flops=n)


# ---- the same in 64 bits -----------------------------------------------------------------------------


def _axis64(nc, ig, o, h):
    """Coarse node coordinates (float, accumulated) and each fine position's cell and offset."""
    gpos = np.zeros(nc, np.float32)
    gpos[0] = o
    for i in range(1, nc):
        gpos[i] = np.float32(float(gpos[i - 1]) + h * ig[i - 1])
    v = (o + np.arange(1 + sum(ig)) * h).astype(np.float32)
    cell = np.clip(np.searchsorted(gpos, v, side="right"), 1, nc - 1) - 1
    g64 = gpos.astype(np.float64)
    return torch.from_numpy(cell).cuda(), torch.from_numpy((v - g64[cell]) / (g64[cell + 1] - g64[cell])).cuda()


def _interp64(coarse, spec):
    nxc, nyc, nzc, ix, iy, iz, x0, y0, z0, h = spec
    s = 1.0 / coarse.double()
    for dim, (n, ig, o) in ((3, (nxc, ix, x0)), (2, (nyc, iy, y0)), (1, (nzc, iz, z0))):
        cell, f = _axis64(n, ig, o, h)
        f = f.reshape([-1 if d == dim else 1 for d in range(4)])
        s = s.index_select(dim, cell) * (1 - f) + s.index_select(dim, cell + 1) * f
    return 1.0 / s


def _cell64(g, x, y, z, dims):
    """Corner index and offsets of positions (tensors) in the fields' grid."""
    out = []
    for v, o, d, n in ((x, g.x0, g.df, dims[0]), (y, g.y0, g.dq, dims[1]), (z, g.z0, g.h, dims[2])):
        i = ((v - o) / d).to(torch.int64).clamp(0, n - 2)
        out += [i, (v - (o + d * i)) / d]
    return out


def _trilinear(t, c):
    i, fx, j, fy, k, fz = c
    s = 0.0
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                w = (fx if di else 1 - fx) * (fy if dj else 1 - fy) * (fz if dk else 1 - fz)
                s = s + w * t[k + dk, j + dj, i + di].double()
    return s


def _locate64(state):
    """The grid search and its two refinements, statistics and interpolation in 64 bits."""
    g, fields = state["grid"], state["fields"]
    nz, ny, nx = fields[0].shape
    got = {k: [] for k in ("exm", "eym", "ezm", "stdmin", "resmin", "tps")}
    for ob in state["events"]:
        idx = [o[0] for o in ob]
        t0 = torch.tensor([o[1] for o in ob], dtype=torch.float64, device="cuda")
        wt = torch.tensor([o[2] for o in ob], dtype=torch.float64, device="cuda")
        sc = [float(g.vpvs) if g.ivs == 0 and o[3] == "S" else 1.0 for o in ob]
        good = torch.ones(len(ob), dtype=torch.float64, device="cuda")
        ngood, retried = len(ob), False

        def stats(times):
            w = good * wt
            a = r2 = 0.0
            for q, t in enumerate(times):
                res = t0[q] - t
                a, r2 = a + w[q] * res, r2 + w[q] * res * res
            fac = w.sum()
            return ((r2 - a * a / fac) / ((ngood - 4) * fac / ngood)).abs().sqrt(), a / fac

        for _ in range(2 * len(ob) + 4):
            s, _a = stats(fields[i][g.kmin:].double() * sc[q] for q, i in enumerate(idx))
            best = int(s.argmin())
            std = float(s.reshape(-1)[best])
            p = [g.x0 + g.df * (best % nx), g.y0 + g.dq * (best // nx % ny), g.z0 + g.h * (best // (nx * ny) + g.kmin)]
            step = [g.df, g.dq, g.h]
            low = [g.x0, g.y0, g.z0 + g.kmin * g.h]
            top = [g.x0 + (nx - 1) * g.df, g.y0 + (ny - 1) * g.dq, g.z0 + (nz - 1) * g.h]
            for div in (g.ndiv, g.ndiv2):
                ax = []
                for a in range(3):
                    eps = 1e-6 * step[a]
                    lo = max(p[a] - step[a], low[a]) if p[a] - step[a] >= low[a] - eps else p[a]
                    hi = p[a] + step[a]
                    n = int(round((min(hi, top[a]) - lo) / step[a] * div)) + (1 if hi <= top[a] + eps else 0)
                    ax.append(lo + step[a] / div * torch.arange(max(n, 1), dtype=torch.float64, device="cuda"))
                z, y, x = (v.reshape(-1) for v in torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij"))
                c = _cell64(g, x, y, z, (nx, ny, nz))
                s, _a = stats(_trilinear(fields[i], c) * sc[q] for q, i in enumerate(idx))
                b = int(s.argmin())
                if float(s[b]) < std:
                    std, p = float(s[b]), [float(x[b]), float(y[b]), float(z[b])]
                step = [d / div for d in step]
            c = _cell64(g, *(torch.tensor([v], dtype=torch.float64, device="cuda") for v in p), (nx, ny, nz))
            times = torch.cat([_trilinear(fields[i], c) * sc[q] for q, i in enumerate(idx)])
            _s, avr = stats(list(times))
            off = (t0 - times - avr).abs()
            keep = ((off <= g.resthres) | (100.0 * off / times <= g.resthrep)).double()
            now = good * keep
            ngood, redo = int(now.sum()), bool((now != good).any())
            good = now
            if ngood < g.nthres:
                break
            if not redo and not retried:
                retried = True
                redo = bool((keep > good).any())
                good = torch.maximum(good, keep)
                ngood = int(good.sum())
            if not redo:
                break
        for k, v in zip(("exm", "eym", "ezm", "stdmin"), p + [std]):
            got[k].append(v)
        got["resmin"] += (t0 - times).tolist()
        got["tps"] += times.tolist()
    return {k: np.array(v) for k, v in got.items()}


def _rays64(state):
    """The residual and hypocentre derivatives at the event; the rays themselves have no 64-bit form here."""
    g, n, obs = state["grid"], state["n"], state["obs"]
    col = {k: np.array([getattr(obs[i], k) for i in range(n)]) for k in ("ex", "ey", "ez", "obstime", "pwt", "field")}
    dims = (g.nx, g.ny, g.nz)
    stack = torch.stack(state["fields"])
    pos = [torch.from_numpy(col[k]).cuda() for k in ("ex", "ey", "ez")]
    i, fx, j, fy, k, fz = _cell64(g, *pos, dims)
    f = torch.from_numpy(col["field"]).cuda().long()
    t, d = 0.0, [0.0, 0.0, 0.0]
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                v = stack[f, k + dk, j + dj, i + di].double()
                wx, wy, wz = (fx if di else 1 - fx), (fy if dj else 1 - fy), (fz if dk else 1 - fz)
                t = t + wx * wy * wz * v
                d[0] = d[0] + (2 * di - 1) * wy * wz * v / g.df
                d[1] = d[1] + wx * (2 * dj - 1) * wz * v / g.dq
                d[2] = d[2] + wx * wy * (2 * dk - 1) * v / g.h
    wet = torch.from_numpy(np.sqrt(col["pwt"])).cuda()
    am = torch.stack([wet] + [x * wet for x in d], 1)
    return dict(dt=(torch.from_numpy(col["obstime"]).cuda() - t).cpu().numpy(), am=am.cpu().numpy())


def exact(case, seed):
    """c2f, slowness, locations and the rays' residuals in 64 bits.  The solves have none: their result is
    the end of a sequence of up to millions of dependent updates, which takes minutes in plain numpy."""
    if case["op"] not in ("locate", "rays", "c2f", "slowness"):
        return None
    state = prepare(case, seed)
    if case["op"] == "locate":
        return _locate64(state)
    if case["op"] == "rays":
        return _rays64(state)
    if case["op"] == "c2f":
        return _interp64(state["coarse"], state["spec"])
    return 1.0 / state["v"].double()
