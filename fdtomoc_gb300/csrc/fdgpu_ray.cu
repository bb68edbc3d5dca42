/* sphrayderv's per-observation work on the device: residual and hypocentre derivatives at the event,
 * the ray traced back from the event down the travel-time gradient to the station, and the ray's
 * slowness derivatives on the coarse metagrid (reference src/sphrayderv.c:1054-2232,
 * lib/sphrayderv/dfind.c, pmin.c), against travel-time fields already on the device.
 *
 * Two lanes trace a ray: a ray is a chain of dependent cell crossings, and the observations of a run
 * are independent.  Another warp beside them adds the segments to the rays' derivative lists.  Every intermediate keeps the C type the reference gives it (the type
 * decides the rounding), the build has no fused multiply-add contraction, and sin/cos/atan2 are
 * correctly rounded (fd_trig_fx.h, fd_trig.h), so the results are bit-identical to the oracle's
 * double-double mode.  A ray's derivatives go to its own list of (coarse node, value) in the order
 * the segments add them, which gives each node the same float sum the reference's dense array
 * gets.
 *
 * A second kernel packs the lists, by node as the reference scans its array, into the caller's arrays. */
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/fdgpu.h"
#include "fd_trig.h"
#include "fd_trig_fx.h"
#include "fdgpu_device.h"

extern "C" int fdh_ctx_device(const fdgpu_ctx *ctx);
extern "C" void *fdh_ctx_stream(const fdgpu_ctx *ctx);
extern "C" void *fdh_ctx_pool(fdgpu_ctx *ctx);
extern "C" int fdh_ctx_fail(fdgpu_ctx *ctx, int cuda_error, const char *what);

namespace {

constexpr float kRearth = 6371.0f;   /* src/sphrayderv.c:87 */

struct RayGridDev {
    int nx, ny, nz, nxc, nyc, nzc;
    double x0, y0, z0, h, dq, df;
};

struct RayObsDev {
    double ex, ey, ez, xs, ys, zs;
    const float *t;
    float obstime, pwt, tc;
    int out;              /* the observation's index in the caller's arrays */
};

/* sin and cos, atan2: in fixed point where that proves the rounding, else in double-double (the same value).
 * A segment's two sincos and two atan2 were 1000 of its 1500 FP64 instructions; 8192 rays in 201x201x81:
 * 49.1 -> 29.1 ms. */
__device__ __noinline__ void sincos_dd(double x, double *s, double *c)
{
    fdt_dd a, b;
    fdt_sincos_full(x, &a, &b);
    *s = a.hi + a.lo;
    *c = b.hi + b.lo;
}

__device__ __noinline__ double atan2_dd(double y, double x) { return fdt_atan2(y, x); }

__device__ __noinline__ void sincos_rn(double x, double *s, double *c)
{
    if (!fdx_sincos(x, s, c)) sincos_dd(x, s, c);
}

__device__ __noinline__ double atan2_rn(double y, double x)
{
    double a;
    return fdx_atan2(y, x, &a) ? a : atan2_dd(y, x);
}

/* (int) of a double as x86-64 converts it: truncation, INT_MIN for NaN and out-of-range values */
__device__ __forceinline__ int trunc_i(double v)
{
    return ((__double2hiint(v) >> 20) & 2047) >= 1023 + 31 ? INT_MIN : (int)v;
}

/* v < 0, v > 0, v != 0 by the bits: a comparison in FP64 takes as long as a product */
__device__ __forceinline__ bool below0(double v)
{
    const unsigned long long u = __double_as_longlong(v);
    return u > 0x8000000000000000ull && u <= 0xfff0000000000000ull;
}
__device__ __forceinline__ bool above0(double v)
{
    const unsigned long long u = __double_as_longlong(v);
    return u != 0 && u <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool not0(double v) { return __double_as_longlong(v) << 1 != 0; }

/* The distances to a cell's three walls are floats, zero or more, or "none", which the reference writes as the double
 * -1e20 (lib/sphrayderv/pmin.c, dfind.c) and which is kNone here */
constexpr float kNone = -1.f;

__device__ __forceinline__ float pmin(float d1, float d2)
{
    if (d1 >= 0) return (d2 >= 0) ? (d1 < d2 ? d1 : d2) : d1;
    return d2 >= 0 ? d2 : kNone;
}

/* the order of the distances' magnitudes, 1e20 for none */
__device__ __forceinline__ unsigned magnitude(float d)
{
    return d == kNone ? 2u * 0x60ad78ecu - 1u : 2u * (__float_as_uint(d) & 0x7fffffffu);
}

/* tolmin, tolmax: rounded up to float, which compares with floats as the double itself */
__device__ __forceinline__ void dfind(const float dd[3], float *d, int *md, float tolmin, float tolmax)
{
    const unsigned a0 = magnitude(dd[0]), a1 = magnitude(dd[1]), a2 = magnitude(dd[2]);
    const int mn = a0 <= a1 && a0 <= a2 ? 0 : a1 <= a2 ? 1 : 2;
    int mid, mx;
    if (mn == 0) {
        mid = a1 <= a2 ? 1 : 2;
        mx = 3 - mid;
    } else if (mn == 1) {
        mid = a0 <= a2 ? 0 : 2;
        mx = 2 - mid;
    } else {
        mid = a0 <= a1 ? 0 : 1;
        mx = 1 - mid;
    }
    auto at = [&](int q) { return q == 0 ? dd[0] : q == 1 ? dd[1] : dd[2]; };
    int m = mn;
    if (at(mn) < tolmin) {
        if (at(mid) < tolmin) m = at(mx) < tolmax ? mx : mid;
        else if (at(mid) < tolmax) m = mid;
    }
    *d = at(m);
    *md = m;
}

/* the times at the corners of fine cell (ie, je, ke); false if one falls outside the field */
__device__ __forceinline__ bool corners(const RayGridDev &g, const float *t, int ie, int je, int ke, float tv[8])
{
    const long long nxy = (long long)g.nx * g.ny, n = nxy * g.nz;
    const long long at = nxy * ke + (long long)g.nx * je + ie;   /* the smallest index */
    if (at < 0 || at + nxy + g.nx + 1 >= n) return false;
    const float *c = t + at, *c2 = c + nxy;
    tv[0] = c[0];
    tv[1] = c[1];
    tv[2] = c[g.nx];
    tv[3] = c[g.nx + 1];
    tv[4] = c2[0];
    tv[5] = c2[1];
    tv[6] = c2[g.nx];
    tv[7] = c2[g.nx + 1];
    return true;
}

/* sin and cos of the cell-wall angles a ray meets: rows y(j) = dq j + y0 and y(j) + dq, columns
 * x(i) = df i + x0 and x(i) + df, for j in [0, ny], i in [0, nx]; the same double-double functions
 * as everywhere else, so a table entry equals a direct call bit for bit */
struct WallTrig {
    const double4 *row;   /* (sin y, cos y, sin(y + dq), cos(y + dq)) */
    const double4 *col;   /* (sin x, cos x, sin(x + df), cos(x + df)) */
};

__global__ void ray_wall_trig(RayGridDev g, double4 *row, double4 *col)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double4 v;
    if (k <= g.ny) {
        const double yj = g.dq * k + g.y0;
        sincos_rn(yj, &v.x, &v.y);
        sincos_rn(yj + g.dq, &v.z, &v.w);
        row[k] = v;
    }
    if (k <= g.nx) {
        const double xi = g.df * k + g.x0;
        sincos_rn(xi, &v.x, &v.y);
        sincos_rn(xi + g.df, &v.z, &v.w);
        col[k] = v;
    }
}

/* a table's row, or a direct call off the table */
__device__ __forceinline__ double4 walls(const double4 *table, int n, int i, double step, double origin)
{
    if (i >= 0 && i <= n) return table[i];
    const double a = step * i + origin;
    double4 v;
    sincos_rn(a, &v.x, &v.y);
    sincos_rn(a + step, &v.z, &v.w);
    return v;
}

/* A block traces 32 rays: warps 0 and 1 step them, two lanes a ray, and hand the segments through shared memory to
 * warp 2, which adds them to the rays' derivative lists meanwhile, four rays at a time with a lane per corner of the
 * coarse cell.  A round is kRound segments of every ray; the warps change buffers at its end.  With one lane doing
 * both, and sorting its list at the end, the lists took two thirds of the time (scattered searches, and an insertion
 * sort whose lanes wait for the longest): 8192 rays in 201x201x81 24.7 -> 9.7 ms. */
constexpr int kRays = 32, kRound = 8, kRayBlock = 96;
constexpr int kMaxCoarse = 8192;   /* coarse coordinates of the three axes */
constexpr int kSeen = 4096;   /* bits of a ray's filter of listed nodes */

struct RaySums {
    float4 seg[2][kRound][kRays];   /* midpoint and length */
    int n[2][kRays];
    /* the ray's list: entries, current coarse cell (i1 = 0: none), and its corners' list positions and sums */
    int len[kRays], over[kRays], i1[kRays], j1[kRays], k1[kRays];
    int pos[kRays][8];
    float sum[kRays][8];
    unsigned seen[kRays][kSeen / 32];
    int nnz[kRays];
};

__device__ __forceinline__ unsigned seen_bit(int node) { return ((unsigned)node * 2654435769u) >> 20; }

/* a segment's length from its record: all are floats but the one that stands for "no wall" */
__device__ __forceinline__ double seg_length(float d) { return d == -1e20f ? -1e20 : (double)d; }

/* in a nondecreasing array: whether cell `at` (at > 0) is the first with v < g[at] */
__device__ __forceinline__ bool coarse_same(const float *g, float v, int at)
{
    return at > 0 && v < g[at] && (at == 1 || v >= g[at - 1]);
}

/* the first q >= 1 with v < g[q]; the lanes of a group of eight search together */
__device__ __forceinline__ int coarse_cell(const float *g, int n, float v, unsigned group, int q)
{
    for (int e = 1; e < n; e += 8) {
        const unsigned hit = __ballot_sync(group, e + q < n && v < g[min(e + q, n - 1)]) & group;
        if (hit) return e + ((__ffs(hit) - 1) & 7);
    }
    return 1;   /* not reached: the tracer ends a ray whose midpoint has no cell */
}

/* Warp 2: adds buffer `buf` to the lists.  A ray crosses several fine cells per coarse cell, and every segment in
 * one coarse cell adds to the same eight nodes: the lanes keep their sums.  On entering the next cell the
 * nodes that it shares with the last one come from the neighbour lanes; the others are new unless the filter
 * has seen them (4 % of the time by chance), when the list is searched. */
__device__ __forceinline__ void add_segments(const RayGridDev &g, const float *gx, const float *gy, const float *gz, bool sorted,
                                             RaySums &sh, int buf, const int *out, int nrays, int cap, int *lidx, float *lval)
{
    const int lane = threadIdx.x & 31, q = lane & 7;
    const unsigned group = 0xffu << (lane & 24);
    const int nxyc = g.nxc * g.nyc, nxyzc = nxyc * g.nzc;
    for (int r0 = 0; r0 < nrays; r0 += 4) {
        const int r = r0 + (lane >> 3), n = r < nrays ? sh.n[buf][r] : 0;
        const int steps = __reduce_max_sync(0xffffffffu, n);
        if (steps == 0) continue;
        int *li = lidx + (size_t)out[r] * cap;
        float *lv = lval + (size_t)out[r] * cap;
        int i1 = sh.i1[r], j1 = sh.j1[r], k1 = sh.k1[r], pos = sh.pos[r][q], len = sh.len[r], over = sh.over[r];
        float sum = sh.sum[r][q];
        for (int s = 0; s < steps; s++) {
            const bool has = s < n;
            const float4 m = has ? sh.seg[buf][s][r] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (has && !(sorted && coarse_same(gx, m.x, i1) && coarse_same(gy, m.y, j1) && coarse_same(gz, m.z, k1))) {
                const int i = coarse_cell(gx, g.nxc, m.x, group, q);
                const int j = coarse_cell(gy, g.nyc, m.y, group, q);
                const int k = coarse_cell(gz, g.nzc, m.z, group, q);
                if (i != i1 || j != j1 || k != k1) {
                    /* corner indices start at column i, as the reference writes them (src/sphrayderv.c:2195-2205) */
                    const int bx = q & 1, by = (q >> 1) & 1, bz = q >> 2;
                    const int node = nxyc * (k - 1 + bz) + g.nxc * (j - 1 + by) + i + bx;
                    if (i1 && pos >= 0) lv[pos] = sum;
                    /* this corner seen from the last cell */
                    const int ox = bx + i - i1, oy = by + j - j1, oz = bz + k - k1;
                    const bool shared = i1 && (ox >> 1) == 0 && (oy >> 1) == 0 && (oz >> 1) == 0;
                    const int from = shared ? (lane & 24) + ox + 2 * oy + 4 * oz : lane;
                    const int opos = __shfl_sync(group, pos, from);
                    const float osum = __shfl_sync(group, sum, from);
                    const bool use = node < nxyzc;
                    unsigned *seen = sh.seen[r];
                    const unsigned bit = use ? seen_bit(node) : 0;
                    const bool look = use && !(shared && opos >= 0) && ((seen[bit >> 5] >> (bit & 31)) & 1u);
                    pos = shared && use ? opos : -1;
                    sum = osum;
                    unsigned want = __ballot_sync(group, look) & group;
                    __syncwarp(group);   /* the sums above are written */
                    while (want) {
                        const int l = __ffs(want) - 1, key = __shfl_sync(group, node, l);
                        want &= want - 1;
                        int at = -1;
                        for (int e = q; e < len; e += 8)
                            if (li[e] == key) at = e;
                        const unsigned hit = __ballot_sync(group, at >= 0) & group;
                        if (!hit) continue;
                        at = __shfl_sync(group, at, __ffs(hit) - 1);
                        if (lane == l) {
                            pos = at;
                            sum = lv[at];
                        }
                    }
                    /* the rest are appended, in corner order */
                    const bool fresh = use && pos < 0;
                    const unsigned add = __ballot_sync(group, fresh) & group;
                    if (fresh) {
                        const int at = len + __popc(add & ((1u << lane) - 1));
                        sum = 0.f;
                        if (at < cap) {
                            pos = at;
                            li[at] = node;
                            atomicOr(&seen[bit >> 5], 1u << (bit & 31));
                        }
                    }
                    len = min(cap, len + __popc(add));
                    if (!use) pos = -2;
                    __syncwarp(group);
                    i1 = i;
                    j1 = j;
                    k1 = k;
                }
            }
            __syncwarp();
            if (has) {
                const double fx = (m.x - gx[i1 - 1]) / (gx[i1] - gx[i1 - 1]);
                const double fy = (m.y - gy[j1 - 1]) / (gy[j1] - gy[j1 - 1]);
                const double fz = (m.z - gz[k1 - 1]) / (gz[k1] - gz[k1 - 1]);
                const float ds = (q & 4 ? fz : 1.f - fz) * (q & 2 ? fy : 1.f - fy) * (q & 1 ? fx : 1.f - fx);
                const double v = ds * seg_length(m.w);
                if (pos >= 0) sum = (float)((double)sum + v);
                over |= pos == -1;
            }
            __syncwarp();
        }
        over = (__ballot_sync(0xffffffffu, over) & group) != 0;
        if (n) {
            sh.pos[r][q] = pos;
            sh.sum[r][q] = sum;
        }
        if (n && q == 0) {
            sh.i1[r] = i1;
            sh.j1[r] = j1;
            sh.k1[r] = k1;
            sh.len[r] = len;
            sh.over[r] = over;
        }
    }
}

/* the largest of g[1..n): a value has a coarse cell if it is below one of them */
__device__ __forceinline__ float coarse_end(const float *g, int n)
{
    float m = -INFINITY;
    for (int q = 1; q < n; q++) m = fmaxf(m, g[q]);
    return m;
}

__device__ __forceinline__ double other(double v) { return __shfl_xor_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float other(float v) { return __shfl_xor_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ int other(int v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

/* Warps 0 and 1: the rays.  A segment is a chain of some 430 FP64 instructions, each of which takes its scheduler 64
 * cycles for one lane as for 32, and of 1800 others for its two sincos and two atan2.  The two lanes of a ray hold the
 * same state; where two of the chain's steps are the same operation on other operands (longitude and colatitude,
 * the two sines of a gradient's denominators, the wall of constant colatitude and that of constant radius,
 * whose equation has a = 1) each lane takes one, and they exchange the results: `second` is the lane's role.  Idle
 * pairs step along on harmless values, without jumps, so that every exchange is one of whole warps.
 * 8192 rays in 201x201x81: 9.5 -> 6.0 ms against a ray a lane. */
__device__ __forceinline__ void trace_rays(const RayGridDev &g, const WallTrig &wt, const float *gx, const float *gy, const float *gz,
                                           RaySums &sh, const RayObsDev *obs, int nrays, int max_seg, fdgpu_ray_result &r)
{
    const int ray = threadIdx.x >> 1;
    const bool second = threadIdx.x & 1, mine = ray < nrays;
    const RayObsDev ob = obs[mine ? ray : 0];
    const float xend = coarse_end(gx, g.nxc), yend = coarse_end(gy, g.nyc), zend = coarse_end(gz, g.nzc);
    const float *t = ob.t;
    const double x0 = g.x0, y0 = g.y0, z0 = g.z0, h = g.h, dq = g.dq, df = g.df;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const float tolmin = __double2float_ru(h * 1.E-6f), tolmax = __double2float_ru(h * 6.0f);
    const double hmil = h / 1000.f, df4 = 4 * df, dq4 = 4 * dq, h4 = 4 * h;
    const float hmilf = __double2float_ru(hmil);
    const double xs = ob.xs, ys = ob.ys, zs = ob.zs;
    const int is = (int)round((xs - x0) / df), js = (int)round((ys - y0) / dq), ks = (int)round((zs - z0) / h);
    const int iscell = trunc_i((xs - x0) / df), jscell = trunc_i((ys - y0) / dq), kscell = trunc_i((zs - z0) / h);
    const double ex = ob.ex, ey = ob.ey, ez = ob.ez;
    const int ies = trunc_i((ex - x0) / df), jes = trunc_i((ey - y0) / dq), kes = trunc_i((ez - z0) / h);
    const float xis = df * ies + x0, yjs = dq * jes + y0, zks = h * kes + z0;

    double xx = ex, yy = ey, zz = ez;
    int ie = ies, je = jes, ke = kes;
    int nseg = 0;
    bool live = false;
    float x2, y2, z2;   /* the station in the cartesian frame, for the last cells (src/sphrayderv.c:1812-1817) */
    do {
        if (!mine) break;
        float tc8[8];
        if (!corners(g, t, ie, je, ke, tc8)) { r.status = FDGPU_RAY_OUTSIDE; break; }
        bool notime = false;
        for (int q = 0; q < 8; q++) notime = notime || tc8[q] > 1.E9;
        if (notime) { r.status = FDGPU_RAY_NOTIME; break; }

        /* residual and hypocentre derivatives at the event (src/sphrayderv.c:1366-1441) */
        {
            const double fx = (xx - xis) / df, fy = (yy - yjs) / dq, fz = (zz - zks) / h;
            float ds[8];
            ds[0] = (1.f - fz) * (1.f - fy) * (1.f - fx);
            ds[1] = (1.f - fz) * (1.f - fy) * fx;
            ds[2] = (1.f - fz) * fy * (1.f - fx);
            ds[3] = (1.f - fz) * fy * fx;
            ds[4] = fz * (1.f - fy) * (1.f - fx);
            ds[5] = fz * (1.f - fy) * fx;
            ds[6] = fz * fy * (1.f - fx);
            ds[7] = fz * fy * fx;
            double dt = 0;
            for (int q = 0; q < 8; q++) dt += ds[q] * tc8[q];
            dt += 0.0f;
            dt += ob.tc;
            dt = ob.obstime - dt;
            r.dt = dt;
            r.resmin = (float)dt;
            float dsdx[8], dsdy[8], dsdz[8];
            dsdx[0] = -(1.f - fz) * (1.f - fy);
            dsdx[1] = (1.f - fz) * (1.f - fy);
            dsdx[2] = -(1.f - fz) * fy;
            dsdx[3] = (1.f - fz) * fy;
            dsdx[4] = -fz * (1.f - fy);
            dsdx[5] = fz * (1.f - fy);
            dsdx[6] = -fz * fy;
            dsdx[7] = fz * fy;
            dsdy[0] = -(1.f - fz) * (1.f - fx);
            dsdy[1] = -(1.f - fz) * fx;
            dsdy[2] = (1.f - fz) * (1.f - fx);
            dsdy[3] = (1.f - fz) * fx;
            dsdy[4] = -fz * (1.f - fx);
            dsdy[5] = -fz * fx;
            dsdy[6] = fz * (1.f - fx);
            dsdy[7] = fz * fx;
            dsdz[0] = -(1.f - fy) * (1.f - fx);
            dsdz[1] = -(1.f - fy) * fx;
            dsdz[2] = -fy * (1.f - fx);
            dsdz[3] = -fy * fx;
            dsdz[4] = (1.f - fy) * (1.f - fx);
            dsdz[5] = (1.f - fy) * fx;
            dsdz[6] = fy * (1.f - fx);
            dsdz[7] = fy * fx;
            float dtdx = 0, dtdy = 0, dtdz = 0;
            for (int q = 0; q < 8; q++) {
                dtdx += dsdx[q] * tc8[q];
                dtdy += dsdy[q] * tc8[q];
                dtdz += dsdz[q] * tc8[q];
            }
            dtdx /= df;
            dtdy /= dq;
            dtdz /= h;
            const float wet = sqrtf(ob.pwt);
            r.wet = wet;
            r.am[0] = wet;
            r.am[1] = dtdx * wet;
            r.am[2] = dtdy * wet;
            r.am[3] = dtdz * wet;
        }

        {
            const double rr = kRearth - zs;
            double sxs, cxs, sys_, cys;
            sincos_rn(xs, &sxs, &cxs);
            sincos_rn(ys, &sys_, &cys);
            x2 = rr * sys_ * cxs;
            y2 = rr * sys_ * sxs;
            z2 = rr * cys;
        }

        live = true;
    } while (false);

    /* the ray (src/sphrayderv.c:1444-2232) */
    int iseg = 0, isegm1 = 0, isegm2 = 0;
    for (int buf = 0;; buf ^= 1) {
        int count = 0;
        for (int step = 0; step < kRound && __any_sync(0xffffffffu, live); step++) {
            if (!live) {
                xx = yy = 1.;
                zz = 0.;
                ie = je = ke = 0;
            }
            const double zk = h * ke + z0;
            double sn, cs;
            sincos_rn(second ? xx : yy, &sn, &cs);
            const double sno = other(sn), cso = other(cs);
            const double sinq = second ? sno : sn, cosq = second ? cso : cs;
            const double sinf_ = second ? sn : sno, cosf_ = second ? cs : cso;

            /* the distance to the station: the last segment in its cell or this near to it */
            const float du = (second ? xx : yy) - (second ? xs : ys), dzs = zz - zs;
            const float rs = kRearth - zz;
            const float dfs1 = rs * sinq * du, dqs1 = rs * du;
            const float part = second ? dfs1 : dqs1, parto = other(part);
            const float dfs = second ? part : parto, dqs = second ? parto : part;
            const float dlen = sqrtf(dfs * dfs + dqs * dqs + dzs * dzs);
            const bool last = live && ((ie == iscell && je == jscell && ke == kscell) || dlen < hmilf);
            if (last) {
                const float mu = (second ? xx : yy) - du * 0.5f, zm = zz - dzs * 0.5f;
                const unsigned pair = 3u << (threadIdx.x & 30);
                const bool in = (second ? mu < xend : mu < yend) && zm < zend;
                if (__all_sync(pair, in)) {
                    float4 &m = sh.seg[buf][count][ray];
                    if (second) {
                        m.x = mu;
                    } else {
                        m.y = mu;
                        m.z = zm;
                        m.w = dlen;
                    }
                    count++;
                    r.status = FDGPU_RAY_OK;
                } else {
                    r.status = FDGPU_RAY_COARSE;
                }
            }
            __syncwarp();
            bool go = live && !last;
            float tv[8] = {0.f, 1.f, 2.f, 4.f, 8.f, 16.f, 32.f, 64.f};
            if (go && nseg >= max_seg) {
                go = false;
                r.status = FDGPU_RAY_STEPS;
            }
            if (go && !corners(g, t, ie, je, ke, tv)) {
                go = false;
                r.status = FDGPU_RAY_OUTSIDE;
            }

            /* the gradient */
            const double r1 = kRearth - zk, r2 = r1 - h;
            const double4 rw = walls(wt.row, g.ny, je, dq, y0), cw = walls(wt.col, g.nx, ie, df, x0);
            const double sqm = second ? rw.z : rw.x;
            const double lo = (second ? tv[3] - tv[2] : tv[1] - tv[0]) / (r1 * sqm);
            const double hi = (second ? tv[7] - tv[6] : tv[5] - tv[4]) / (r2 * sqm);
            const double fq = (second ? tv[6] + tv[7] - tv[4] - tv[5] : tv[2] + tv[3] - tv[0] - tv[1]) / (second ? r2 : r1);
            const double loo = other(lo), hio = other(hi), fqo = other(fq);
            const double sum0 = lo + loo + hi + hio, sum1 = fqo + fq;   /* the first lane's, the second's */
            const double gd = -((second ? sum1 : sum0) / (second ? dq4 : df4)), gdo = other(gd);
            double g0 = second ? gdo : gd, g1 = second ? gd : gdo;
            double g2 = (tv[4] + tv[5] + tv[6] + tv[7] - tv[0] - tv[1] - tv[2] - tv[3]) / h4;

            /* the direction */
            const double ro = kRearth - zz;
            const double xo = ro * sinq * cosf_, yo = ro * sinq * sinf_, zo = ro * cosq;
            const double gm = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
            const double gu = (second ? g1 : g0) / gm, guo = other(gu);
            const double sf = second ? guo : gu, sq = second ? gu : guo, sr = g2 / gm;
            const double u1 = second ? cosf_ : -sinf_, u2 = second ? sinf_ : cosf_;
            double su = u1 * sf + cosq * u2 * sq + sinq * u2 * sr, suo = other(su);
            double sz = -sinq * sq + cosq * sr;
            {
                const double ax = second ? suo : su, ay = second ? su : suo;
                const float smag = sqrtf((float)(ax * ax + ay * ay + sz * sz));
                su /= smag;
                sz /= smag;
            }
            suo = other(su);
            double sx = second ? suo : su, sy = second ? su : suo;
            if (ie >= (is - 2) && ie < (is + 2) && je >= (js - 2) && je < (js + 2) && ke >= (ks - 2) && ke < (ks + 2)) {
                const double dx = x2 - xo, dy = y2 - yo, dz = z2 - zo;
                const double dl = sqrt(dx * dx + dy * dy + dz * dz);
                sx = dx / dl;
                sy = dy / dl;
                sz = dz / dl;
            }
            __syncwarp();

            /* the walls: the first lane takes radius and longitude, the second colatitude */
            const bool near0 = second ? below0(g1) : below0(g0);
            const double sinw = second ? (near0 ? rw.x : rw.z) : (near0 ? cw.x : cw.z);
            const double cosw = second ? (near0 ? rw.y : rw.w) : (near0 ? cw.y : cw.w);
            const bool big = fabs(cosw) > fabs(sinw);
            const double tn = (big ? sinw : cosw) / (big ? cosw : sinw), tn2 = tn * tn;
            const double m1 = second && !big ? tn2 : 1., m2 = second ? (big ? tn2 : 1.) : -1.;
            const double rwall = above0(g2) ? r1 : r2;
            const double a = second ? (sx * sx + sy * sy) * m1 - sz * sz * m2 : 1.;
            const double b = (xo * sx + yo * sy) * m1 - zo * sz * m2;
            const double c = (xo * xo + yo * yo) * m1 - zo * zo * m2 - (second ? 0. : rwall * rwall);
            const double quad = b * b - a * c, root = sqrt(quad);
            const double n1 = -b + root, n2 = -b - root;
            const double lin = big ? xo * tn - yo : yo * tn - xo, lden = big ? sy - sx * tn : sx - sy * tn;
            const float v1 = (second ? n1 : lin) / (second ? a : lden);
            const float v2 = n2 / a;
            float du_ = kNone, dl_ = kNone;
            if (not0(second ? g1 : g2) && quad >= 0) du_ = pmin(second ? v1 : (float)n1, v2);
            if (not0(g0) && v1 > 0) dl_ = v1;   /* the first lane's */
            const float duo = other(du_);
            float dd[3] = {__shfl_sync(0xffffffffu, dl_, threadIdx.x & 30), second ? du_ : duo, second ? duo : du_};

            const int back3 = iseg + isegm1 + isegm2;
            if (below0(g0)) {
                if (dd[0] < hmilf && (iseg == 1 || (back3 == 1 && nseg >= 3))) { g0 = 0.; dd[0] = kNone; }
            } else if (above0(g0)) {
                if (dd[0] < hmilf && (iseg == -1 || (back3 == -1 && nseg >= 3))) { g0 = 0; dd[0] = kNone; }
            } else {
                dd[0] = kNone;
            }
            if (below0(g1)) {
                if (dd[1] < hmilf && (iseg == 20 || (back3 == 20 && nseg >= 3))) { g1 = 0.; dd[1] = kNone; }
            } else if (above0(g1)) {
                if (dd[1] < hmilf && (iseg == -20 || (back3 == -20 && nseg >= 3))) { g1 = 0; dd[1] = kNone; }
            } else {
                dd[1] = kNone;
            }
            if (above0(g2)) {
                if (dd[2] < hmilf && (iseg == 300 || (back3 == 300 && nseg >= 3))) { g2 = 0.; dd[2] = kNone; }
            } else if (below0(g2)) {
                if (dd[2] < hmilf && (iseg == -300 || (back3 == -300 && nseg >= 3))) { g2 = 0; dd[2] = kNone; }
            } else {
                dd[2] = kNone;
            }

            float dist;
            int md;
            dfind(dd, &dist, &md, tolmin, tolmax);
            const double d = dist == kNone ? -1e20 : (double)dist;

            /* the next point */
            const double pu = (second ? yo : xo) + d * (second ? sy : sx), puo = other(pu), zn = zo + d * sz;
            const double xn = second ? puo : pu, yn = second ? pu : puo;
            const double h2 = xn * xn + yn * yn;
            const double rt = sqrt(second ? h2 : h2 + zn * zn);
            const double ang = atan2_rn(second ? rt : yn, second ? zn : xn), ango = other(ang);
            const double xnew = second ? ango : ang, ynew = second ? ang : ango;
            const double znew = kRearth - __shfl_sync(0xffffffffu, rt, threadIdx.x & 30);
            const float mu = ((second ? ynew : xnew) + (second ? yy : xx)) * 0.5, zm = (znew + zz) * 0.5;
            /* its cell: the two coordinates that no wall gives */
            const bool byq = second ? md == 2 : md == 0;
            const double cu = byq ? ynew - y0 : second ? znew - z0 : xnew - x0;
            const int cell = trunc_i(cu / (byq ? dq : second ? h : df)), cello = other(cell);
            const int ca = second ? cello : cell, cb = second ? cell : cello;
            const bool in = (second ? mu < yend : mu < xend) && zm < zend;
            const bool inside = other((int)in) && in;
            if (go) {
                xx = xnew;
                yy = ynew;
                zz = znew;
                nseg++;
                isegm2 = isegm1;
                isegm1 = iseg;
                bool left = false;
                if (md == 0) {
                    je = ca;
                    ke = cb;
                    if (below0(g0)) {
                        if (ie < 0) left = true; else { ie--; iseg = -1; }
                    } else {
                        if (ie >= nx - 1) left = true; else { ie++; iseg = 1; }
                    }
                } else if (md == 1) {
                    if (below0(g1)) {
                        if (je < 0) left = true; else { je--; iseg = -20; }
                    } else {
                        if (je >= ny - 1) left = true; else { je++; iseg = 20; }
                    }
                    ie = ca;
                    ke = cb;
                } else {
                    if (above0(g2)) {
                        if (ke < 0) left = true; else { ke--; iseg = -300; }
                    } else {
                        if (ke >= nz - 1) left = true; else { ke++; iseg = 300; }
                    }
                    ie = ca;
                    je = cb;
                }
                if (left || (xx < x0 || ie >= nx) || (yy < y0 || je >= ny) || (zz < z0 || ke >= nz)) {
                    r.status = FDGPU_RAY_LEFT;
                    go = false;
                } else if (!inside) {
                    r.status = FDGPU_RAY_COARSE;
                    go = false;
                } else {
                    float4 &m = sh.seg[buf][count][ray];
                    if (second) {
                        m.y = mu;
                    } else {
                        m.x = mu;
                        m.z = zm;
                        m.w = (float)d;
                    }
                    count++;
                }
            }
            live = go;
            __syncwarp();
        }
        if (!second) sh.n[buf][ray] = count;
        if (__syncthreads_and(!live)) break;   /* the buffer to the last warp */
    }
    r.nseg = nseg;
}

__global__ void __launch_bounds__(kRayBlock) ray_trace(RayGridDev g, WallTrig wt, const float *__restrict__ coarse,
                                                       const RayObsDev *__restrict__ obs, int nobs, int max_seg,
                                                       int cap, fdgpu_ray_result *__restrict__ res,
                                                       int *__restrict__ nlist, int *__restrict__ lidx, float *__restrict__ lval)
{
    extern __shared__ float s_coarse[];
    __shared__ RaySums sh;
    __shared__ int out[kRays];
    const int ncoarse = g.nxc + g.nyc + g.nzc;
    const int first = blockIdx.x * kRays, nrays = min(kRays, nobs - first);
    const float *gx = s_coarse, *gy = s_coarse + g.nxc, *gz = s_coarse + g.nxc + g.nyc;
    for (int q = threadIdx.x; q < ncoarse; q += blockDim.x) s_coarse[q] = coarse[q];
    for (int q = threadIdx.x; q < kRays * (kSeen / 32); q += blockDim.x) sh.seen[q / (kSeen / 32)][q % (kSeen / 32)] = 0;
    if (threadIdx.x < kRays) {
        const int r = threadIdx.x;
        out[r] = r < nrays ? obs[first + r].out : 0;
        sh.len[r] = sh.over[r] = sh.i1[r] = sh.j1[r] = sh.k1[r] = 0;
        for (int q = 0; q < 8; q++) sh.pos[r][q] = -2;
    }
    __syncthreads();
    bool sorted = true;
    for (int q = threadIdx.x; q < ncoarse - 1; q += blockDim.x)
        if (q != g.nxc - 1 && q != g.nxc + g.nyc - 1 && !(s_coarse[q] <= s_coarse[q + 1])) sorted = false;
    sorted = __syncthreads_and(sorted);
    fdgpu_ray_result r;
    memset(&r, 0, sizeof r);
    if (threadIdx.x < 2 * kRays) {
        trace_rays(g, wt, gx, gy, gz, sh, obs + first, nrays, max_seg, r);
    } else {
        for (int b = 0;; b ^= 1) {
            const bool last = __syncthreads_and(1);   /* buffer b is full; whether every ray has ended */
            add_segments(g, gx, gy, gz, sorted, sh, b, out, nrays, cap, lidx, lval);
            if (last) break;
        }
        __syncwarp();
        for (int e = threadIdx.x & 31; e < 8 * nrays; e += 32)
            if (sh.pos[e >> 3][e & 7] >= 0) lval[(size_t)out[e >> 3] * cap + sh.pos[e >> 3][e & 7]] = sh.sum[e >> 3][e & 7];
    }
    __syncthreads();
    for (int q = threadIdx.x >> 5; q < nrays; q += kRayBlock / 32) {
        int nz = 0;
        for (int e = threadIdx.x & 31; e < sh.len[q]; e += 32) nz += lval[(size_t)out[q] * cap + e] != 0;
        nz = __reduce_add_sync(0xffffffffu, nz);
        if ((threadIdx.x & 31) == 0) sh.nnz[q] = nz;
    }
    __syncthreads();
    if (threadIdx.x < 2 * nrays && !(threadIdx.x & 1)) {
        const int q = threadIdx.x >> 1;
        if (r.status == FDGPU_RAY_OK && sh.over[q]) r.status = FDGPU_RAY_STEPS;
        r.nnz = r.status == FDGPU_RAY_OK ? sh.nnz[q] : 0;
        nlist[out[q]] = sh.len[q];
        res[out[q]] = r;
    }
}

/* The rays' lists into the packed arrays, a warp per ray: ascending node order, zero sums dropped
 * (src/sphrayderv.c:1548-1552).  An entry's place is the number of nonzero entries with smaller nodes: n^2/32
 * comparisons side by side, 0.04 ms for 8192 rays' 1.6 million entries. */
__global__ void ray_pack(const fdgpu_ray_result *__restrict__ res, const long long *__restrict__ off,
                         const int *__restrict__ nlist, int nobs, int cap, const int *__restrict__ lidx,
                         const float *__restrict__ lval, int *__restrict__ idx, float *__restrict__ du)
{
    const int w = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (w >= nobs || res[w].nnz == 0) return;
    const int n = nlist[w];
    const long long base = off[w];
    const int *li = lidx + (size_t)w * cap;
    const float *lv = lval + (size_t)w * cap;
    for (int e0 = 0; e0 < n; e0 += 32) {
        const int e = e0 + lane, key = e < n ? li[e] : 0;
        const float v = e < n ? lv[e] : 0.f;
        int at = 0;
        for (int f0 = 0; f0 < n; f0 += 32) {
            const int f = f0 + lane;
            const int other = f < n && lv[f] != 0 ? li[f] : INT_MAX;
#pragma unroll 8
            for (int q = 0; q < 32; q++) at += __shfl_sync(0xffffffffu, other, q) < key;
        }
        if (v != 0) {
            idx[base + at] = key;
            du[base + at] = v;
        }
    }
}

}  // namespace

#define RAY_CU(call)                                                        \
    do {                                                                    \
        const cudaError_t e_ = (call);                                      \
        if (e_ != cudaSuccess) return fdh_ctx_fail(ctx, (int)e_, #call);    \
    } while (0)

extern "C" int fdgpu_ray_default_limits(const fdgpu_ray_grid *g, int *max_seg, int *cap)
{
    if (!g) return FDGPU_EINVAL;
    if (max_seg) *max_seg = 16 * (g->nx + g->ny + g->nz) + 256;
    if (cap) *cap = 8 * (g->nx + g->ny + g->nz) + 64;
    return FDGPU_OK;
}

extern "C" int fdgpu_raytrace(fdgpu_ctx *ctx, const fdgpu_ray_grid *g, const float *const *d_fields, int nfields,
                              int nobs, const fdgpu_ray_obs *obs, int max_seg, int cap, fdgpu_ray_result *res,
                              long long *off, int *idx, float *du, long long total_cap, void *stream)
{
    if (!ctx || !g || nobs < 0 || nobs > (1 << 24) || (nobs > 0 && (!d_fields || !obs || !res || !off)))
        return FDGPU_EINVAL;
    if (g->nx < 2 || g->ny < 2 || g->nz < 2 || g->nxc < 2 || g->nyc < 2 || g->nzc < 2 || !g->gx || !g->gy || !g->gz
        || !(g->h > 0) || !(g->dq > 0) || !(g->df > 0))
        return FDGPU_EINVAL;
    if ((long long)g->nx * g->ny * g->nz >= (1ll << 31) || (long long)g->nxc * g->nyc * g->nzc >= (1ll << 30)
        || g->nxc + g->nyc + g->nzc > kMaxCoarse)
        return FDGPU_EINVAL;
    int dseg = 0, dcap = 0;
    fdgpu_ray_default_limits(g, &dseg, &dcap);
    if (max_seg <= 0) max_seg = dseg;
    if (cap <= 0) cap = dcap;
    for (int k = 0; k < nobs; k++)
        if (obs[k].field < 0 || obs[k].field >= nfields || !d_fields[obs[k].field]) return FDGPU_EINVAL;
    off[0] = 0;
    if (nobs == 0) return FDGPU_OK;
    FdDeviceScope dev_(fdh_ctx_device(ctx));
    if (dev_.err) return FDGPU_ENODEV;
    cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)fdh_ctx_stream(ctx);

    /* launch order: longest rays first (cells between event and station), so that a warp's rays end
     * together; each result goes back to its observation's slot */
    std::vector<int> order(nobs);
    std::vector<double> span(nobs);
    for (int k = 0; k < nobs; k++) {
        const fdgpu_ray_obs &o = obs[k];
        span[k] = std::fabs((o.ex - o.xs) / g->df) + std::fabs((o.ey - o.ys) / g->dq) + std::fabs((o.ez - o.zs) / g->h);
        if (!(span[k] == span[k])) span[k] = 0;
        order[k] = k;
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return span[a] > span[b]; });
    std::vector<RayObsDev> hobs(nobs);
    for (int q = 0; q < nobs; q++) {
        const fdgpu_ray_obs &o = obs[order[q]];
        hobs[q] = RayObsDev{o.ex, o.ey, o.ez, o.xs, o.ys, o.zs, d_fields[o.field], o.obstime, o.pwt, o.tc, order[q]};
    }
    const int ncoarse = g->nxc + g->nyc + g->nzc;
    std::vector<float> hc(ncoarse);
    std::memcpy(hc.data(), g->gx, sizeof(float) * g->nxc);
    std::memcpy(hc.data() + g->nxc, g->gy, sizeof(float) * g->nyc);
    std::memcpy(hc.data() + g->nxc + g->nyc, g->gz, sizeof(float) * g->nzc);

    FdArena mem(fdh_ctx_pool(ctx), st);
    RayObsDev *dobs;
    float *dcoarse, *lval, *ddu;
    int *lidx, *didx, *dn;
    fdgpu_ray_result *dres;
    long long *doff;
    double4 *drow, *dcol;
    RAY_CU(mem.get(&dobs, nobs));
    RAY_CU(mem.get(&drow, (size_t)g->ny + 1));
    RAY_CU(mem.get(&dcol, (size_t)g->nx + 1));
    RAY_CU(mem.get(&dcoarse, ncoarse));
    RAY_CU(mem.get(&dres, nobs));
    RAY_CU(mem.get(&dn, nobs));
    RAY_CU(mem.get(&lidx, (size_t)nobs * cap));
    RAY_CU(mem.get(&lval, (size_t)nobs * cap));
    RAY_CU(mem.get(&doff, nobs + 1));
    RAY_CU(cudaMemcpyAsync(dobs, hobs.data(), sizeof(RayObsDev) * nobs, cudaMemcpyHostToDevice, st));
    RAY_CU(cudaMemcpyAsync(dcoarse, hc.data(), sizeof(float) * ncoarse, cudaMemcpyHostToDevice, st));
    const RayGridDev G{g->nx, g->ny, g->nz, g->nxc, g->nyc, g->nzc, g->x0, g->y0, g->z0, g->h, g->dq, g->df};
    const int nwall = (g->nx > g->ny ? g->nx : g->ny) + 1;
    ray_wall_trig<<<(nwall + 127) / 128, 128, 0, st>>>(G, drow, dcol);
    RAY_CU(cudaGetLastError());
    /* beside the block's own arrays the coarse coordinates (up to 32 KB) pass the 48 KB that need no asking */
    RAY_CU(cudaFuncSetAttribute(ray_trace, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxCoarse * (int)sizeof(float)));
    ray_trace<<<(nobs + kRays - 1) / kRays, kRayBlock, sizeof(float) * ncoarse, st>>>(
        G, WallTrig{drow, dcol}, dcoarse, dobs, nobs, max_seg, cap, dres, dn, lidx, lval);
    RAY_CU(cudaGetLastError());
    RAY_CU(cudaMemcpyAsync(res, dres, sizeof(fdgpu_ray_result) * nobs, cudaMemcpyDeviceToHost, st));
    RAY_CU(cudaStreamSynchronize(st));
    for (int k = 0; k < nobs; k++) off[k + 1] = off[k] + res[k].nnz;
    const long long total = off[nobs];
    if (total > total_cap || (total > 0 && (!idx || !du))) return FDGPU_ETOOBIG;
    if (total == 0) return FDGPU_OK;
    RAY_CU(mem.get(&didx, (size_t)total));
    RAY_CU(mem.get(&ddu, (size_t)total));
    RAY_CU(cudaMemcpyAsync(doff, off, sizeof(long long) * (nobs + 1), cudaMemcpyHostToDevice, st));
    ray_pack<<<(nobs + 7) / 8, 256, 0, st>>>(dres, doff, dn, nobs, cap, lidx, lval, didx, ddu);
    RAY_CU(cudaGetLastError());
    RAY_CU(cudaMemcpyAsync(idx, didx, sizeof(int) * total, cudaMemcpyDeviceToHost, st));
    RAY_CU(cudaMemcpyAsync(du, ddu, sizeof(float) * total, cudaMemcpyDeviceToHost, st));
    RAY_CU(cudaStreamSynchronize(st));
    return FDGPU_OK;
}
