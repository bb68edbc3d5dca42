/*
 * fdgpu_locate.cu — event location on device-resident travel-time fields: the grid search of
 * FDtomoC's sphfdloc (reference src/sphfdloc.c), for many events per call, with results
 * bit-identical to the reference's.
 *
 * Per event the reference runs (a) a coarse search over the grid nodes from depth index kmin
 * (:729-794), (b) a refinement with ndiv steps per cell around the best node (:840-895), (c) a second
 * refinement with ndiv2 steps per first-refinement step around the best point (:967-1056), each
 * trial point scored by the standard deviation of its weighted residuals, then (d) drops outliers or
 * recovers phases and repeats (a)-(c) if that changed the phase set (:1086-1128).
 *
 * GPU form: a thread keeps the reference's sequential per-phase accumulation of its trial points, every
 * event of the batch in the same launch, so the statistics match bit for bit; the "first strictly smaller" scan over trial points becomes an atomicMin on
 * (float bits of the deviation << 32 | trial index in loop order), which picks the same point.  A
 * kernel between stages takes the minimum, updates the event's best point the
 * way the sequential scan would, and lays out the next stage's window; a last one recomputes the
 * residuals at the final point and runs the outlier / recovery step.  The host repeats the stages
 * for the events that asked for another pass.
 *
 * Refinements.  The reference interpolates each phase's time in double and rounds the residual to float:
 * 26 FP64 instructions a phase and trial, which held the FP64 units (2 lanes a clock on an SM) 86 % busy.
 * Here the residual along a row of trials is A - b f in pairs of floats (about 46 bits), A and b formed once per
 * row, cell and phase; its float is certain unless the value lies within the pairs' error of
 * a rounding boundary (fd_pair.h), and only such residuals are formed in double.
 * The floats that enter the statistics are the reference's either way.
 *
 * Arithmetic: statistics in float, positions and trilinear weights in double, as the reference;
 * compiled with --fmad=false and IEEE float division and square root.  At grid nodes the residual
 * obstime - t of two floats is formed in float: the reference forms it in double and rounds to
 * float, and the two agree for all finite floats (when the exponents differ by 29 or less the double
 * difference is exact, so one rounding happens in both; beyond that the smaller operand is below a
 * half unit of the larger and both give the larger).
 */
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "fd_pair.h"
#include "fdgpu.h"
#include "fdgpu_device.h"

namespace {

constexpr int kLocBlock = 256;
constexpr int kMaxObs = 800;   /* the reference's maxobs (include/common/parameter.h) */

enum { kActive = 0, kAccepted = 1, kTooFew = 2, kStdHigh = 3, kRedo = 4 };

struct LocEvent {
    int obs0, nobs;
    int ngood, iretry, passes, state;
    float stdmin, avrmin;
    int nxx, nyy, nzz;
    int wstage;                 /* stage of the last new minimum: 0 coarse, 1, 2 */
    double exm, eym, ezm;
    double x0i, y0i, z0i, sx, sy, sz;   /* current refinement window: origin and steps */
    int nsx, nsy, nsz;
    int nlist;                  /* accepted phases of this pass, listed from obs0 on */
    float facs;                 /* their weights' sum, in phase order (the same at every trial point) */
    unsigned long long best;    /* (deviation bits << 32) | trial index; ~0: none */
};

struct LocObsDev {
    const float *field;
    float obstime, pwt;
    int s_scaled;   /* S phase whose time is the P field times vpvs (ivs 0) */
};

/* a trial coordinate along one axis of an event's window: its cell and its place in the cell, as find_cell
 * forms it, and that place as a pair of floats */
struct AxisPos {
    double f;
    float fh, fl;
    int cell;
};

__device__ __forceinline__ unsigned long long trial_key(float std, unsigned idx)
{
    /* only deviations that can win: finite (the running minimum starts at +inf, and NaN never
     * compares smaller) */
    if (!(std < INFINITY)) return ~0ull;
    return ((unsigned long long)__float_as_uint(std) << 32) | idx;
}

/* The cell containing (x, yy, z), clamped to the grid, and its eight trilinear weights, as find_time
 * forms them (:1305-1345).  All fields share the grid, so a trial point computes these once for all
 * its phases; each weight is the same product, in the same order, that the reference multiplies by
 * the corner's time. */
struct Cell {
    long long a, b, a2, b2;
    int i;
    double w[8];
};

__device__ __forceinline__ void cell_weights(Cell &c, double fx, double fy, double fz)
{
    c.w[0] = (1.0 - fx) * (1.0 - fy) * (1.0 - fz);
    c.w[1] = fx * (1.0 - fy) * (1.0 - fz);
    c.w[2] = (1.0 - fx) * fy * (1.0 - fz);
    c.w[3] = (1.0 - fx) * (1.0 - fy) * fz;
    c.w[4] = fx * fy * (1.0 - fz);
    c.w[5] = fx * (1.0 - fy) * fz;
    c.w[6] = (1.0 - fx) * fy * fz;
    c.w[7] = fx * fy * fz;
}

/* the cell of coordinate x on an axis of n nodes at o + d i, clamped to the grid, and x's place in it */
__device__ __forceinline__ int axis_cell(double x, double o, double d, int n, double *f)
{
    int i = (int)((x - o) / d);
    i = i < 0 ? 0 : i;
    i = i > n - 2 ? n - 2 : i;
    *f = (x - (o + d * i)) / d;
    return i;
}

__device__ __forceinline__ void find_cell(const fdgpu_loc_grid &g, double x, double yy, double z, Cell &c)
{
    double fx, fy, fz;
    const int i = axis_cell(x, g.x0, g.df, g.nx, &fx), j = axis_cell(yy, g.y0, g.dq, g.ny, &fy);
    const int k = axis_cell(z, g.z0, g.h, g.nz, &fz);
    c.a = (long long)g.nx * g.ny * k;
    c.b = (long long)g.nx * j;
    c.a2 = (long long)g.nx * g.ny * (k + 1);
    c.b2 = (long long)g.nx * (j + 1);
    c.i = i;
    cell_weights(c, fx, fy, fz);
}

/* the trilinear time of one field in that cell: the reference's sum, term by term */
__device__ __forceinline__ double cell_time(const Cell &c, const float *t)
{
    const int i = c.i;
    double tp = c.w[0] * (double)t[c.a + c.b + i];
    tp = tp + c.w[1] * (double)t[c.a + c.b + i + 1];
    tp = tp + c.w[2] * (double)t[c.a + c.b2 + i];
    tp = tp + c.w[3] * (double)t[c.a2 + c.b + i];
    tp = tp + c.w[4] * (double)t[c.a + c.b2 + i + 1];
    tp = tp + c.w[5] * (double)t[c.a2 + c.b + i + 1];
    tp = tp + c.w[6] * (double)t[c.a2 + c.b2 + i];
    tp = tp + c.w[7] * (double)t[c.a2 + c.b2 + i + 1];
    return tp;
}

/* one phase's residual at a trial point whose time is tp (double) */
__device__ __forceinline__ float residual_d(const LocObsDev &o, double tp, float vpvs)
{
    if (o.s_scaled) tp *= (double)vpvs;
    return (float)((double)o.obstime - tp);
}

/* the accumulation of :750-770 for one accepted phase (facs: LocEvent) */
__device__ __forceinline__ void accumulate(float res, float wt, float &avres, float &rsq)
{
    const float r1 = res * wt;
    const float r2 = r1 * res;
    avres += r1;
    rsq += r2;
}

/* :771-777 */
__device__ __forceinline__ float deviation(float avres, float rsq, float facs, int ngood)
{
    const float avwt = facs / (float)ngood;
    const float deb = (rsq - avres * avres / facs) / ((float)(ngood - 4) * avwt);
    return sqrtf(fabsf(deb));
}

/* Whether a trial's deviation is certainly above the smallest one found so far, `best` (any earlier value of the
 * event's minimum serves).  It is formed without the divisions and the square root of deviation(), within
 * 2^-20 rsq / den of its square; NaN and infinite values answer no.
 * Almost every trial ends here: two divisions and a square root cost as much as the sums of several phases. */
struct Hopeless {
    float rf, rd, b2;
    __device__ __forceinline__ Hopeless(float facs, int ngood, unsigned long long best)
    {
        const float b = __uint_as_float((unsigned)(best >> 32));
        rf = 1.0f / facs;
        rd = 1.0f / ((float)(ngood - 4) * (facs / (float)ngood));
        b2 = best == ~0ull ? INFINITY : b * b * 1.00000191f + 1e-36f;
    }
    __device__ __forceinline__ bool operator()(float avres, float rsq) const
    {
        const float q = rsq * rd;
        return (rsq - avres * avres * rf) * rd - 1.9073486e-06f * fabsf(q) > b2;
    }
};

__device__ __forceinline__ unsigned long long load_best(const LocEvent &ev)
{
    return *const_cast<const volatile unsigned long long *>(&ev.best);
}

/* the block's smallest key into the event's minimum */
__device__ __forceinline__ void reduce_key(unsigned long long key, unsigned long long *dst)
{
    __shared__ unsigned long long red[kLocBlock / 32];
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
        key = other < key ? other : key;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = key;
    __syncthreads();
    if (threadIdx.x < 32) {
        key = threadIdx.x < kLocBlock / 32 ? red[threadIdx.x] : ~0ull;
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
            key = other < key ? other : key;
        }
        if (threadIdx.x == 0 && key != ~0ull) atomicMin(dst, key);
    }
}

/* obstime - t * vpvs as the reference forms it (in double, then float) */
__device__ __noinline__ float residual_scaled(float obstime, float t, float vpvs)
{
    return (float)((double)obstime - (double)t * (double)vpvs);
}

/* the same in pairs of floats, which nearly always tell (fd_pair.h) */
__device__ __forceinline__ float residual_scaled_pair(float obstime, float t, float vpvs)
{
    float res;
    return fdp_scaled_residual(obstime, t, vpvs, &res) ? res : residual_scaled(obstime, t, vpvs);
}

/* a phase as the coarse search reads it from shared memory, in one 16-byte load */
struct __align__(16) CoarseObs {
    const float *field;   /* at the block's first node */
    float obstime, pwt;
};

/* the statistics of nodes n .. n+3 over the event's accepted phases */
template <bool SCALED>
__device__ __forceinline__ void coarse_sums(const CoarseObs *ob, const unsigned char *scaled, int nl, int at, bool wide, int left,
                                            float vpvs, float av[4], float rs[4])
{
    constexpr int kBatch = 4;   /* phases whose loads are in flight together */
    auto load = [&](const CoarseObs &o) {
        const float *f = o.field + at;
        if (wide) return __ldg(reinterpret_cast<const float4 *>(f));
        return make_float4(f[0], left > 1 ? f[1] : 0.f, left > 2 ? f[2] : 0.f, left > 3 ? f[3] : 0.f);
    };
    auto add = [&](const CoarseObs &o, int q, const float4 &tv) {
        const float t[4] = {tv.x, tv.y, tv.z, tv.w};
        const bool sc = SCALED && scaled[q];
#pragma unroll
        for (int i = 0; i < 4; i++) accumulate(sc ? residual_scaled_pair(o.obstime, t[i], vpvs) : o.obstime - t[i], o.pwt, av[i], rs[i]);
    };
    int q = 0;
    for (; q + kBatch <= nl; q += kBatch) {
        CoarseObs o[kBatch];
        float4 tv[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            o[u] = ob[q + u];
            tv[u] = load(o[u]);
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) add(o[u], q + u, tv[u]);
    }
    for (; q < nl; q++) {
        const CoarseObs o = ob[q];
        add(o, q, load(o));
    }
}

/* (a) Coarse search: trial c is grid node n0 + c, in the reference's loop order.  What bounds it is reading a
 * time per phase and node, and five float operations on it.  A thread takes four nodes, one 16-byte load per
 * phase, and consecutive blocks take the same nodes for successive events, so that the events of a catalog,
 * which share their stations' fields, find them in L2.  128 events x 32 phases on 201x201x81: 10.5 -> 4.7 ms a
 * pass against a node a thread with the events one after another (52 GB of DRAM reads, 0.8 GB now). */
__global__ void __launch_bounds__(kLocBlock) loc_coarse(fdgpu_loc_grid g, const LocObsDev *list, LocEvent *evs,
                                                          const int *active, int nact, long long n0, long long n1,
                                                          int aligned)
{
    __shared__ CoarseObs ob[kMaxObs];
    __shared__ unsigned char scaled[kMaxObs];
    LocEvent &ev = evs[active[blockIdx.x % (unsigned)nact]];
    const int nl = ev.nlist;
    /* nodes first + 4 threadIdx.x ..; the first group may begin before n0, the last end after n1 */
    const long long first = (n0 & ~3ll) + 4ll * (blockIdx.x / (unsigned)nact) * kLocBlock;
    bool any = false;
    for (int q = threadIdx.x; q < nl; q += blockDim.x) {
        const LocObsDev o = list[ev.obs0 + q];
        ob[q] = CoarseObs{o.field + first, o.obstime, o.pwt};
        scaled[q] = (unsigned char)o.s_scaled;
        any = any || o.s_scaled;
    }
    any = __syncthreads_or(any);
    const unsigned long long best = load_best(ev);
    const int at = 4 * threadIdx.x;
    const long long n = first + at;
    unsigned long long key = ~0ull;
    if (n < n1) {
        float av[4] = {0.f, 0.f, 0.f, 0.f}, rs[4] = {0.f, 0.f, 0.f, 0.f};
        const int left = n1 - n > 4 ? 4 : (int)(n1 - n);
        if (any) coarse_sums<true>(ob, scaled, nl, at, aligned && left > 3, left, g.vpvs, av, rs);
        else coarse_sums<false>(ob, scaled, nl, at, aligned && left > 3, left, g.vpvs, av, rs);
        const Hopeless hopeless(ev.facs, ev.ngood, best);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (n + i < n0 || i >= left || hopeless(av[i], rs[i])) continue;
            const unsigned long long k = trial_key(deviation(av[i], rs[i], ev.facs, ev.ngood), (unsigned)(n + i - n0));
            key = k < key ? k : key;
        }
    }
    reduce_key(key, &ev.best);
}

/* one phase's residual at place (fx,fy,fz) of the cell with corner times at t: the reference's (find_time) */
__device__ __noinline__ float residual_exact(const LocObsDev &o, const float *t, int nx, int nxy, double fx, double fy,
                                             double fz, float vpvs)
{
    Cell c;
    c.a = 0;
    c.b = 0;
    c.a2 = nxy;
    c.b2 = nx;
    c.i = 0;
    cell_weights(c, fx, fy, fz);
    return residual_d(o, cell_time(c, t), vpvs);
}

/* (b), (c) refinements: trial c = (k * nsy + j) * nsx + i of the event's window (header comment).  A block's
 * consecutive trials lie on a few rows (j, k) and in at most three cells of each (segments); the phases go
 * through in tiles whose coefficients, a pair of floats for a and b and the margin m per segment, fit shared
 * memory.
 *
 * Residuals that are not certain.  Where the places in a cell are fractions of few bits (8 or 16 divisions) every tenth
 * residual is a tie of two floats, and where times fit well the residuals are small and the margin a larger part of
 * their last place.  Formed where they occur, one such residual costs its warp the 43 FP64 instructions of all 32
 * lanes.  So a tile's uncertain residuals are listed, formed with full warps, and handed back before the sums.
 * First and second refinement of 128 events x 32 phases, against FP64 throughout and against forming them where they
 * occur: 41^3 trials 15.3 and 15.2 -> 2.03 and 0.58 -> 0.99 and 0.65 ms; 17^3 trials (8 divisions, scaled S) 1.20
 * and 1.20 -> 1.41 and 0.24 -> 0.25 and 0.10. */
constexpr int kTile = 12;     /* phases of a tile at most, their residuals in registers: with 16 four blocks no longer fit an SM */
constexpr int kCoef = 1024;   /* coefficients of a tile: segments x phases */
constexpr int kFix = 1024;    /* uncertain residuals formed together; with more a tile takes several rounds */
constexpr int kDivMax = 64;   /* largest divisions of the axis tables; finer windows take loc_refine_fp64 */
static_assert(kLocBlock <= 256 && kTile <= 256 && kTile <= kFix, "entries of the list: phase << 8 | thread");

__global__ void __launch_bounds__(kLocBlock, 4) loc_refine(fdgpu_loc_grid g, const LocObsDev *list, LocEvent *evs,
                                                          const int *active, const AxisPos *axes, int naxis)
{
    __shared__ fdp_row cab[kCoef];
    __shared__ float cm[kCoef];
    __shared__ fdp_ff wrow[kLocBlock + 2][4];
    __shared__ int orow[kLocBlock + 2];
    __shared__ float fixv[kFix];
    __shared__ unsigned short fixq[kFix];
    __shared__ int nfix;
    constexpr unsigned kNone = 0xffffu;
    const int e = active[blockIdx.y];
    LocEvent &ev = evs[e];
    const int nsx = ev.nsx, nsy = ev.nsy, ncand = nsx * nsy * ev.nsz;
    const int c0 = blockIdx.x * kLocBlock;
    if (c0 >= ncand) return;
    const AxisPos *ax = axes + (size_t)e * 3 * naxis, *ay = ax + naxis, *az = ay + naxis;
    const LocObsDev *ob = list + ev.obs0;
    const int nl = ev.nlist, nx = g.nx, nxy = g.nx * g.ny;
    const int c = c0 + threadIdx.x, clast = min(c0 + kLocBlock, ncand) - 1;
    const int row0 = c0 / nsx, nrows = clast / nsx - row0 + 1;
    const int cmin = ax[0].cell, ncx = ax[nsx - 1].cell - cmin + 1;
    const int segs = nrows * ncx, tile = min(kTile, kCoef / segs);
    for (int r = threadIdx.x; r < nrows; r += kLocBlock) {
        const int row = row0 + r, k = row / nsy, j = row - k * nsy;
        fdp_weights(fdp_pair(ay[j].fh, ay[j].fl), fdp_pair(az[k].fh, az[k].fl), wrow[r]);
        orow[r] = az[k].cell * nxy + ay[j].cell * nx;
    }
    float avres = 0.0f, rsq = 0.0f, fh = 0.f, fl = 0.f;
    int seg = 0;
    if (c < ncand) {
        const int row = c / nsx, i = c - row * nsx;
        fh = ax[i].fh;
        fl = ax[i].fl;
        seg = (row - row0) * ncx + ax[i].cell - cmin;
    }
    for (int q0 = 0; q0 < nl; q0 += tile) {
        const int nq = min(tile, nl - q0);
        __syncthreads();
        for (int x = threadIdx.x; x < nq * segs; x += kLocBlock) {
            const int q = x / segs, sg = x - q * segs, r = sg / ncx;
            const LocObsDev o = ob[q0 + q];
            fdp_coefficients(o.obstime, o.s_scaled, g.vpvs, o.field + orow[r] + cmin + (sg - r * ncx), nx, nxy, wrow[r], &cab[x], &cm[x]);
        }
        __syncthreads();
        float res[kTile];
        unsigned open = 0;   /* phases whose residual is not certain */
#pragma unroll
        for (int q = 0; q < kTile; q++)
            if (q < nq && !fdp_residual(&cab[q * segs + seg], cm[q * segs + seg], fh, fl, &res[q])) open |= 1u << q;
        if (c >= ncand) open = 0;
        while (__syncthreads_or(open != 0)) {
            if (threadIdx.x == 0) nfix = 0;
            __syncthreads();
            int at = 0;
            bool fits = false;
            if (open) {
                at = atomicAdd(&nfix, __popc(open));
                fits = at + __popc(open) <= kFix;
                int to = at;
                for (unsigned b = open; b && to < kFix; b &= b - 1) fixq[to++] = (unsigned short)(fits ? (__ffs(b) - 1) << 8 | threadIdx.x : kNone);
            }
            __syncthreads();
            const int n = min(nfix, kFix);
            for (int x = threadIdx.x; x < n; x += kLocBlock) {
                const unsigned it = fixq[x];
                if (it == kNone) continue;
                const LocObsDev &o = ob[q0 + (it >> 8)];
                const int cc = c0 + (int)(it & 255u), row = cc / nsx, k = row / nsy;
                const AxisPos &px = ax[cc - row * nsx];
                fixv[x] = residual_exact(o, o.field + orow[row - row0] + px.cell, nx, nxy, px.f, ay[row - k * nsy].f, az[k].f, g.vpvs);
            }
            __syncthreads();
            if (fits) {
#pragma unroll
                for (int q = 0; q < kTile; q++)
                    if ((open >> q) & 1u) res[q] = fixv[at++];
                open = 0;
            }
        }
#pragma unroll
        for (int q = 0; q < kTile; q++)
            if (q < nq) accumulate(res[q], ob[q0 + q].pwt, avres, rsq);
    }
    unsigned long long key = ~0ull;
    if (c < ncand) key = trial_key(deviation(avres, rsq, ev.facs, ev.ngood), (unsigned)c);
    reduce_key(key, &ev.best);
}

/* the refinements in double throughout, for windows finer than the axis tables hold */
__global__ void __launch_bounds__(kLocBlock) loc_refine_fp64(fdgpu_loc_grid g, const LocObsDev *list, LocEvent *evs,
                                                               const int *active)
{
    LocEvent &ev = evs[active[blockIdx.y]];
    const long long ncand = (long long)ev.nsx * ev.nsy * ev.nsz;
    if ((long long)blockIdx.x * kLocBlock >= ncand) return;
    const LocObsDev *ob = list + ev.obs0;
    const long long c = (long long)blockIdx.x * kLocBlock + threadIdx.x;
    unsigned long long key = ~0ull;
    if (c < ncand) {
        const int i = (int)(c % ev.nsx), j = (int)((c / ev.nsx) % ev.nsy), k = (int)(c / ((long long)ev.nsx * ev.nsy));
        const double zp = ev.z0i + ev.sz * k, yp = ev.y0i + ev.sy * j, xp = ev.x0i + ev.sx * i;
        Cell cell;
        find_cell(g, xp, yp, zp, cell);
        float avres = 0.0f, rsq = 0.0f;
        for (int q = 0; q < ev.nlist; q++) accumulate(residual_d(ob[q], cell_time(cell, ob[q].field), g.vpvs), ob[q].pwt, avres, rsq);
        key = trial_key(deviation(avres, rsq, ev.facs, ev.ngood), (unsigned)c);
    }
    reduce_key(key, &ev.best);
}

/* Take the stage's minimum (stage 0 coarse, 1, 2) and lay out the next window. */
__device__ void plan_stage(const fdgpu_loc_grid &g, LocEvent &ev, int stage)
{
    const unsigned long long key = ev.best;
    ev.best = ~0ull;
    const float std = __uint_as_float((unsigned)(key >> 32));
    const unsigned idx = (unsigned)key;
    if (stage == 0) {
        ev.nxx = ev.nyy = ev.nzz = 0;
        ev.stdmin = INFINITY;
        ev.wstage = 0;
        if (key != ~0ull) {
            const long long n = (long long)g.nx * g.ny * g.kmin + idx;
            ev.nxx = (int)(n % g.nx);
            ev.nyy = (int)((n / g.nx) % g.ny);
            ev.nzz = (int)(n / ((long long)g.nx * g.ny));
            ev.stdmin = std;
        }
        ev.exm = g.x0 + ev.nxx * g.df;
        ev.eym = g.y0 + ev.nyy * g.dq;
        ev.ezm = g.z0 + ev.nzz * g.h;
        /* first refinement window (:840-877) */
        const int n1 = g.ndiv + 1, n2 = n1 + g.ndiv;
        int iz0 = ev.nzz - 1, nsz = n2;
        if (iz0 < g.kmin) { iz0 = ev.nzz; nsz = n1; }
        if (ev.nzz == g.nz - 1) nsz = n1 - 1;
        int iy0 = ev.nyy - 1, nsy = n2;
        if (iy0 < 0) { iy0 = ev.nyy; nsy = n1; }
        if (ev.nyy == g.ny - 1) nsy = n1 - 1;
        int ix0 = ev.nxx - 1, nsx = n2;
        if (ix0 < 0) { ix0 = ev.nxx; nsx = n1; }
        if (ev.nxx == g.nx - 1) nsx = n1 - 1;
        ev.z0i = g.z0 + g.h * iz0;
        ev.y0i = g.y0 + g.dq * iy0;
        ev.x0i = g.x0 + g.df * ix0;
        ev.sz = g.h / g.ndiv;
        ev.sy = g.dq / g.ndiv;
        ev.sx = g.df / g.ndiv;
        ev.nsx = nsx;
        ev.nsy = nsy;
        ev.nsz = nsz;
        return;
    }
    if (key != ~0ull && std < ev.stdmin) {
        const int i = (int)(idx % (unsigned)ev.nsx), j = (int)((idx / (unsigned)ev.nsx) % (unsigned)ev.nsy);
        const int k = (int)(idx / ((unsigned)ev.nsx * (unsigned)ev.nsy));
        ev.nxx = i;
        ev.nyy = j;
        ev.nzz = k;
        ev.ezm = ev.z0i + ev.sz * k;
        ev.eym = ev.y0i + ev.sy * j;
        ev.exm = ev.x0i + ev.sx * i;
        ev.stdmin = std;
        ev.wstage = stage;
    }
    if (stage == 1) {
        /* second refinement window (:967-999) */
        const double dh = g.h / g.ndiv, ddq = g.dq / g.ndiv, ddf = g.df / g.ndiv;
        const int n1 = g.ndiv2 + 1, n2 = n1 + g.ndiv2;
        double z0i = ev.ezm - dh;
        int nsz = n2;
        if (z0i <= g.z0 + g.kmin * g.h) { z0i = ev.ezm; nsz = n1; }
        if (ev.ezm + dh > (double)g.zmax) nsz = n1 - 1;
        double y0i = ev.eym - ddq;
        int nsy = n2;
        if (y0i <= g.y0) { y0i = ev.eym; nsy = n1; }
        if (ev.eym + ddq > (double)g.ymax) nsy = n1 - 1;
        double x0i = ev.exm - ddf;
        int nsx = n2;
        if (x0i <= g.x0) { x0i = ev.exm; nsx = n1; }
        if (ev.exm + ddf > (double)g.xmax) nsx = n1 - 1;
        ev.z0i = z0i;
        ev.y0i = y0i;
        ev.x0i = x0i;
        ev.sz = dh / g.ndiv2;
        ev.sy = ddq / g.ndiv2;
        ev.sx = ddf / g.ndiv2;
        ev.nsx = nsx;
        ev.nsy = nsy;
        ev.nsz = nsz;
    }
}

/* A block per event: the stage's minimum and the next window, then (axes given) the window's coordinates along
 * each axis, whose cells and places in them every trial of the window shares. */
__global__ void loc_plan(fdgpu_loc_grid g, LocEvent *evs, const int *active, int stage, AxisPos *axes, int naxis)
{
    const int e = active[blockIdx.x];
    __shared__ LocEvent ev;
    if (threadIdx.x == 0) {
        ev = evs[e];
        plan_stage(g, ev, stage);
        evs[e] = ev;
    }
    __syncthreads();
    if (!axes) return;
    AxisPos *at = axes + (size_t)e * 3 * naxis;
    for (int t = threadIdx.x; t < 3 * naxis; t += blockDim.x) {
        const int axis = t / naxis, i = t - axis * naxis;
        AxisPos p;
        if (axis == 0) p.cell = axis_cell(ev.x0i + ev.sx * i, g.x0, g.df, g.nx, &p.f);
        else if (axis == 1) p.cell = axis_cell(ev.y0i + ev.sy * i, g.y0, g.dq, g.ny, &p.f);
        else p.cell = axis_cell(ev.z0i + ev.sz * i, g.z0, g.h, g.nz, &p.f);
        p.fh = (float)p.f;
        p.fl = (float)(p.f - (double)p.fh);
        at[t] = p;
    }
}

/* Residuals at the final point, then the outlier / recovery step (:1086-1128).  A warp per event: a lane
 * per phase, sums in phase order. */
__global__ void loc_finish(fdgpu_loc_grid g, const LocObsDev *obs, unsigned char *good, LocEvent *evs,
                           const int *active, int nact, float *resmin, float *tps)
{
    const int a = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (a >= nact) return;
    LocEvent &ev = evs[active[a]];
    const bool found = ev.stdmin < INFINITY;
    const int obs0 = ev.obs0, nobs = ev.nobs, wstage = ev.wstage, iretry = ev.iretry;
    const long long node = (long long)g.nx * g.ny * ev.nzz + (long long)g.nx * ev.nyy + ev.nxx;
    float avres = 0.0f;
    Cell cell;
    if (wstage != 0) find_cell(g, ev.exm, ev.eym, ev.ezm, cell);
    for (int q0 = 0; q0 < nobs; q0 += 32) {
        const int o = obs0 + q0 + lane;
        float r1 = 0.f;
        bool in = false;
        if (q0 + lane < nobs) {
            const LocObsDev d = obs[o];
            float res;
            if (wstage == 0)
                res = d.s_scaled ? residual_scaled(d.obstime, d.field[node], g.vpvs) : d.obstime - d.field[node];
            else
                res = residual_d(d, cell_time(cell, d.field), g.vpvs);
            in = good[o] != 0;
            r1 = res * d.pwt;
            /* where no trial became the minimum in this pass the reference keeps the previous pass's
             * values (zero before the first) */
            if (found) {
                resmin[o] = res;
                tps[o] = d.obstime - res;
            }
        }
        for (unsigned b = __ballot_sync(0xffffffffu, in); b; b &= b - 1) avres += __shfl_sync(0xffffffffu, r1, __ffs(b) - 1);
    }
    const float avrmin = found ? avres / ev.facs : 0.0f;
    /* a phase whose residual is off by too much is dropped; on the second look, one dropped before whose
     * residual has come in is taken back */
    int ngood = 0;
    bool redo = false;
    for (int look = 0; look < 2; look++) {
        for (int q0 = 0; q0 < nobs; q0 += 32) {
            const int o = obs0 + q0 + lane;
            bool kept = false, changed = false;
            if (q0 + lane < nobs && (good[o] != 0) == (look == 0)) {
                const float absres = fabsf(resmin[o] - avrmin);
                const float perc = 100.0f * absres / tps[o];
                const bool near = absres <= g.resthres || perc <= g.resthrep;
                kept = near;
                changed = near != (look == 0);
                if (changed) good[o] = look == 0 ? 0 : 1;
            }
            ngood += __popc(__ballot_sync(0xffffffffu, kept));
            redo = __any_sync(0xffffffffu, changed) || redo;
        }
        if (look == 0 && (ngood < g.nthres || redo || iretry >= 1)) break;
        if (look == 0 && lane == 0) ev.iretry = iretry + 1;
    }
    if (lane == 0) {
        ev.avrmin = avrmin;
        ev.ngood = ngood;
        ev.state = ngood < g.nthres ? kTooFew : redo ? kRedo : ev.stdmin <= g.stdmax ? kAccepted : kStdHigh;
    }
}

__global__ void loc_init(LocEvent *evs, const int *offs, int nev)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nev) return;
    LocEvent &ev = evs[e];
    ev.obs0 = offs[e];
    ev.nobs = offs[e + 1] - offs[e];
    ev.ngood = ev.nobs;   /* :686: every phase, flagged or not, before the first check */
    ev.iretry = 0;
    ev.passes = 0;
    ev.state = kActive;
    ev.best = ~0ull;
}

/* A warp per event: its state for the pass, and the phases accepted so far, listed in order. */
__global__ void loc_begin_pass(LocEvent *evs, const int *active, int nact, const LocObsDev *obs, const unsigned char *good,
                               LocObsDev *list)
{
    const int a = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (a >= nact) return;
    LocEvent &ev = evs[active[a]];
    const int obs0 = ev.obs0, nobs = ev.nobs;
    int nl = 0;
    float facs = 0.0f;
    for (int q0 = 0; q0 < nobs; q0 += 32) {
        const int o = obs0 + q0 + lane;
        const bool in = q0 + lane < nobs && good[o] != 0;
        LocObsDev d{};
        if (in) d = obs[o];
        unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) list[obs0 + nl + __popc(b & ((1u << lane) - 1u))] = d;
        nl += __popc(b);
        for (; b; b &= b - 1) facs += __shfl_sync(0xffffffffu, d.pwt, __ffs(b) - 1);
    }
    if (lane == 0) {
        ev.nlist = nl;
        ev.facs = facs;
        ev.passes++;
        ev.state = kActive;
        ev.best = ~0ull;
    }
}

__global__ void loc_results(const LocEvent *evs, int nev, fdgpu_loc_result *out)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nev) return;
    const LocEvent &ev = evs[e];
    fdgpu_loc_result r;
    r.status = ev.state == kAccepted ? 0 : ev.state == kTooFew ? 1 : 2;
    r.ngood = ev.ngood;
    r.nxx = ev.nxx;
    r.nyy = ev.nyy;
    r.nzz = ev.nzz;
    r.passes = ev.passes;
    r.exm = ev.exm;
    r.eym = ev.eym;
    r.ezm = ev.ezm;
    r.stdmin = ev.stdmin;
    r.avrmin = ev.avrmin;
    out[e] = r;
}

__global__ void loc_states(const LocEvent *evs, int nev, int *state)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nev) state[e] = evs[e].state;
}

}  // namespace

/* ---- host side -------------------------------------------------------------------------------- */

#include <cmath>
#include <cstring>
#include <vector>

extern "C" int fdh_ctx_device(const fdgpu_ctx *ctx);
extern "C" void *fdh_ctx_stream(const fdgpu_ctx *ctx);
extern "C" void *fdh_ctx_pool(fdgpu_ctx *ctx);
extern "C" int fdh_ctx_fail(fdgpu_ctx *ctx, int cuda_error, const char *what);

namespace {

constexpr double kHpi = 1.570796f;          /* src/sphfdloc.c:74-75: float literals */
constexpr double kDegrad = 0.017453292f;

}  // namespace

extern "C" void fdgpu_loc_grid_from_spec(fdgpu_loc_grid *g, int nx, int ny, int nz, double x0_deg, double y0_deg,
                                         double z0_km, double h_km)
{
    if (!g) return;
    std::memset(g, 0, sizeof *g);
    g->nx = nx;
    g->ny = ny;
    g->nz = nz;
    g->h = h_km;
    g->z0 = z0_km;
    /* WGS84 geocentric colatitude of the north edge and radius of z = 0, as sphfdloc links it
     * (lib/common/geographic_method.c glath; src/sphfdloc.c:384-394) */
    const double ap = 6378137.0, esq = 6.69437978616733379 * 0.001;
    const double lat = y0_deg * kDegrad;
    const double s = std::sin(lat);
    const double hm = -z0_km * 1000.0;
    const double anu = ap / std::sqrt(1.0 - esq * s * s);
    const double x = (anu + hm) * std::cos(lat);
    const double z = ((1.0 - esq) * anu + hm) * s;
    g->z0r = std::sqrt(x * x + z * z) / 1000.0;
    g->y0 = kHpi - std::atan2(z, x);
    g->x0 = x0_deg * kDegrad;
    g->dq = h_km / 6371.0;
    g->df = std::fabs(h_km / (6371.0 * std::sin(g->y0)));
    g->xmax = (float)(g->x0 + (nx - 1) * g->df);
    g->ymax = (float)(g->y0 + (ny - 1) * g->dq);
    g->zmax = (float)(g->z0 + (nz - 1) * g->h);
    g->kmin = 2;
    g->ndiv = 20;
    g->ndiv2 = 20;
    g->ivs = 1;
    g->vpvs = 1.78f;
    g->nthres = 8;
    g->resthres = 0.5f;
    g->resthrep = 5.0f;
    g->stdmax = 15.0f;
}

#define LOC_CU(call)                                                        \
    do {                                                                    \
        const cudaError_t e_ = (call);                                      \
        if (e_ != cudaSuccess) return fdh_ctx_fail(ctx, (int)e_, #call);    \
    } while (0)

extern "C" int fdgpu_locate(fdgpu_ctx *ctx, const fdgpu_loc_grid *g, const float *const *d_fields, int nfields,
                            int nev, const int *obs_offset, fdgpu_loc_obs *obs, float *resmin, float *tps,
                            fdgpu_loc_result *results, void *stream)
{
    if (!ctx || !g || nev < 0 || (nev > 0 && (!d_fields || !obs_offset || !obs || !resmin || !tps || !results)))
        return FDGPU_EINVAL;
    if (nev == 0) return FDGPU_OK;
    if (g->nx < 2 || g->ny < 2 || g->nz < 2 || g->ndiv < 1 || g->ndiv2 < 1 || g->ndiv > 1000 || g->ndiv2 > 1000
        || g->kmin < 0 || !(g->h > 0) || !(g->dq > 0) || !(g->df > 0))
        return FDGPU_EINVAL;
    if ((long long)g->nx * g->ny * g->nz >= (1ll << 31)) return FDGPU_EINVAL;
    if (obs_offset[0] != 0) return FDGPU_EINVAL;
    for (int e = 0; e < nev; e++) {
        const int n = obs_offset[e + 1] - obs_offset[e];
        if (n < 1 || n > kMaxObs) return FDGPU_EINVAL;
    }
    const int nobs = obs_offset[nev];
    for (int k = 0; k < nobs; k++) {
        const fdgpu_loc_obs &o = obs[k];
        if (o.field < 0 || o.field >= nfields || !d_fields[o.field]) return FDGPU_EINVAL;
        if (o.phase != 'P' && o.phase != 'S') return FDGPU_EINVAL;
    }
    FdDeviceScope dev_(fdh_ctx_device(ctx));
    if (dev_.err) return FDGPU_ENODEV;
    cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)fdh_ctx_stream(ctx);

    /* one block goes to the device, phases, active list and offsets, good flags, residuals, times and results, and
     * its part from the flags on comes back: a copy each way */
    auto up16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
    const size_t o_offs = up16(sizeof(LocObsDev) * nobs), o_act = o_offs + up16(sizeof(int) * (nev + 1));
    const size_t o_good = o_act + up16(sizeof(int) * nev), o_res = o_good + up16(nobs);
    const size_t o_tps = o_res + up16(sizeof(float) * nobs), o_out = o_tps + up16(sizeof(float) * nobs);
    const size_t o_end = o_out + sizeof(fdgpu_loc_result) * nev;
    std::vector<char> block(o_end, 0);
    LocObsDev *hobs = reinterpret_cast<LocObsDev *>(block.data());
    unsigned char *hgood = reinterpret_cast<unsigned char *>(block.data() + o_good);
    for (int k = 0; k < nobs; k++) {
        hobs[k].field = d_fields[obs[k].field];
        hobs[k].obstime = obs[k].obstime;
        hobs[k].pwt = obs[k].pwt;
        hobs[k].s_scaled = (g->ivs == 0 && obs[k].phase == 'S') ? 1 : 0;
        hgood[k] = obs[k].good ? 1 : 0;
    }
    std::memcpy(block.data() + o_offs, obs_offset, sizeof(int) * (nev + 1));
    for (int e = 0; e < nev; e++) reinterpret_cast<int *>(block.data() + o_act)[e] = e;
    FdArena mem(fdh_ctx_pool(ctx), st);
    char *dblock;
    LocObsDev *dlist;
    AxisPos *daxes = nullptr;
    LocEvent *devs;
    int *dstate;
    LOC_CU(mem.get(&dblock, o_end));
    LocObsDev *dobs = reinterpret_cast<LocObsDev *>(dblock);
    int *doffs = reinterpret_cast<int *>(dblock + o_offs), *dact = reinterpret_cast<int *>(dblock + o_act);
    unsigned char *dgood = reinterpret_cast<unsigned char *>(dblock + o_good);
    float *dres = reinterpret_cast<float *>(dblock + o_res), *dtps = reinterpret_cast<float *>(dblock + o_tps);
    fdgpu_loc_result *dout = reinterpret_cast<fdgpu_loc_result *>(dblock + o_out);
    LOC_CU(mem.get(&dlist, nobs));
    /* the windows' axis tables (see loc_refine) */
    const int ndmax = g->ndiv > g->ndiv2 ? g->ndiv : g->ndiv2, naxis = 2 * ndmax + 1;
    if (ndmax <= kDivMax) LOC_CU(mem.get(&daxes, (size_t)nev * 3 * naxis));
    LOC_CU(mem.get(&devs, nev));
    LOC_CU(mem.get(&dstate, nev));
    LOC_CU(cudaMemcpyAsync(dblock, block.data(), o_end, cudaMemcpyHostToDevice, st));
    loc_init<<<(nev + 127) / 128, 128, 0, st>>>(devs, doffs, nev);
    LOC_CU(cudaGetLastError());

    const fdgpu_loc_grid G = *g;
    const long long n0 = (long long)g->kmin * g->nx * g->ny, n1 = (long long)g->nz * g->nx * g->ny;
    const long long ncoarse = n0 < n1 ? (n1 - (n0 & ~3ll) + 3) / 4 : 0;   /* threads: four nodes each */
    const long long nwin[2] = {(long long)(2 * g->ndiv + 1) * (2 * g->ndiv + 1) * (2 * g->ndiv + 1),
                               (long long)(2 * g->ndiv2 + 1) * (2 * g->ndiv2 + 1) * (2 * g->ndiv2 + 1)};
    /* 16-byte loads of four nodes need every field on a 16-byte boundary */
    int aligned = 1;
    for (int k = 0; k < nobs; k++)
        if ((reinterpret_cast<uintptr_t>(hobs[k].field) & 15u) != 0) aligned = 0;
    std::vector<int> act(nev), state(nev);
    for (int e = 0; e < nev; e++) act[e] = e;
    for (int pass = 0; !act.empty(); pass++) {
        if (pass > 2 * kMaxObs + 4) return FDGPU_ESCHED;   /* each redo drops or recovers a phase */
        const int nact = (int)act.size();
        if (pass > 0) LOC_CU(cudaMemcpyAsync(dact, act.data(), sizeof(int) * nact, cudaMemcpyHostToDevice, st));
        const int tw = (nact + 3) / 4;   /* a warp per event */
        loc_begin_pass<<<tw, 128, 0, st>>>(devs, dact, nact, dobs, dgood, dlist);
        if (ncoarse > 0) {
            /* blocks of one launch: tiles x events, within the grid's limit of 2^31 - 1 */
            const long long tiles = (ncoarse + kLocBlock - 1) / kLocBlock;
            const long long most = 0x7fffffffll / tiles;
            for (int a0 = 0; a0 < nact;) {
                const int na = (int)(nact - a0 < most ? nact - a0 : most);
                loc_coarse<<<(unsigned)(tiles * na), kLocBlock, 0, st>>>(G, dlist, devs, dact + a0, na, n0, n1, aligned);
                a0 += na;
            }
        }
        loc_plan<<<nact, 128, 0, st>>>(G, devs, dact, 0, daxes, naxis);
        for (int stage = 1; stage <= 2; stage++) {
            /* grid.y carries the events; more than 65535 go in slices */
            for (int a0 = 0; a0 < nact; a0 += 65535) {
                const int na = nact - a0 < 65535 ? nact - a0 : 65535;
                const dim3 grid((unsigned)((nwin[stage - 1] + kLocBlock - 1) / kLocBlock), na);
                if (daxes) loc_refine<<<grid, kLocBlock, 0, st>>>(G, dlist, devs, dact + a0, daxes, naxis);
                else loc_refine_fp64<<<grid, kLocBlock, 0, st>>>(G, dlist, devs, dact + a0);
            }
            loc_plan<<<nact, 128, 0, st>>>(G, devs, dact, stage, stage == 1 ? daxes : nullptr, naxis);
        }
        loc_finish<<<tw, 128, 0, st>>>(G, dobs, dgood, devs, dact, nact, dres, dtps);
        loc_states<<<(nev + 127) / 128, 128, 0, st>>>(devs, nev, dstate);
        LOC_CU(cudaGetLastError());
        LOC_CU(cudaMemcpyAsync(state.data(), dstate, sizeof(int) * nev, cudaMemcpyDeviceToHost, st));
        LOC_CU(cudaStreamSynchronize(st));
        std::vector<int> next;
        for (int e : act)
            if (state[e] == kRedo) next.push_back(e);
        act.swap(next);
    }
    loc_results<<<(nev + 127) / 128, 128, 0, st>>>(devs, nev, dout);
    LOC_CU(cudaGetLastError());
    LOC_CU(cudaMemcpyAsync(hgood, dgood, o_end - o_good, cudaMemcpyDeviceToHost, st));
    LOC_CU(cudaStreamSynchronize(st));
    std::memcpy(results, block.data() + o_out, sizeof(fdgpu_loc_result) * nev);
    std::memcpy(resmin, block.data() + o_res, sizeof(float) * nobs);
    std::memcpy(tps, block.data() + o_tps, sizeof(float) * nobs);
    for (int k = 0; k < nobs; k++) obs[k].good = hgood[k];
    return FDGPU_OK;
}
