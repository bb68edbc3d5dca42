/*
 * fdgpu_kernels.cu — GB300 kernels of the sphfd travel-time solver.
 *
 *   fd_geo_build    builds the geometry tables of one grid geometry (shared by its stations);
 *   fd_solve        one CTA per station: source box, then the expanding-box sweeps of
 *                   src/sphfd.c:1008-5678 with each face walked in dependency order.
 *
 * Face walk.  The reference updates a face's points one at a time in ascending order of the time
 * of their inner-layer neighbour (ties in fill order, src/sphfd.c:1024-1033 and glibc's stable
 * qsort); a point reads its eight in-face neighbours, seeing the new value of those already
 * updated and the old value of the others.  So the face is a DAG: an edge runs from each point to
 * every in-face neighbour with a larger key (time bits, fill index).  Walking it in dependency order —
 * every point whose earlier neighbours are all done may be evaluated, then releases its later
 * neighbours — reproduces the sequential order exactly.  No sort is needed.
 *
 * The one sequential coupling that is not a neighbour relation is the stale (t0,t4) pair of
 * fdsph2d (src/sphfd.c:6116-6121): a point whose first 2-D trial comes before any 3-D / new-edge
 * call of its own reads the pair left by the previous point in sort order.  Such a point is put
 * aside if a 2-D value wins without that pair, and waits for the record of the largest-key earlier
 * point that made a writer call (or the entry pair); bounds on the times still missing keep that wait
 * short (keys_above, exit_floor).  This is rare on most grids (hundreds of points per million).
 *
 * Within a walk the warps of the CTA are independent workers that meet only at shared-memory
 * counters (see "warp workers" below); every wait among them is bounded and ends in an error
 * status, never in a hang.
 */
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include "fdgpu_eval.cuh"
#include "fdgpu_trials.cuh"
#include "fdgpu_bound.cuh"
#include "fdgpu_layout.h"

#define FD_WARPS 12                 /* independent workers per station */
#define FD_BLOCK (FD_WARPS * 32)

/* optional per-phase cycle counters (thread 0, between barriers) for profiling builds */
#ifdef FDGPU_PHASE_TIMERS
#define FD_TIC(v) long long v = clock64()
#define FD_TOC(k, v) \
    do { if ((threadIdx.x & 31) == 0) atomicAdd(reinterpret_cast<unsigned long long *>(&sh.cyc[k]), (unsigned long long)(clock64() - (v))); } while (0)
#else
#define FD_TIC(v) do { } while (0)
#define FD_TOC(k, v) do { } while (0)
#endif
#define FD_HEADTEST 1.e-3

/* rarely called: kept out of the worker loop's code, whose registers and instruction fetches they would cost */
#define FD_COLD __device__ __noinline__

namespace fdk {

/* ---------------------------------------------------------------------------------------------- */
/* geometry tables                                                                                 */

__global__ void fd_geo_build(int nx, int ny, int nz, double h, double dq, double df, double z0r,
                             const double *ysin, double *zrow, double *node, double *cell)
{
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const double hsq = h * h, dqsq = dq * dq, dfsq = df * df;
    const double is_h = 1.0 / (h * h);
    for (long long z = tid; z < nz; z += stride) {
        const double r = z0r - h * (double)z;  /* rc(z), src/sphfd.c:154 */
        zrow[z * FD_Z_N + FD_Z_R] = r;
        zrow[z * FD_Z_N + FD_Z_RDQ] = r * dq;
        zrow[z * FD_Z_N + FD_Z_INV_RDQ] = 1.0 / (r * dq);
    }
    for (long long k = tid; k < (long long)nz * ny; k += stride) {
        const int z = (int)(k / ny), y = (int)(k % ny);
        const double r = z0r - h * (double)z, s = ysin[y];
        const double rsdf = (r * s) * df, rdq = r * dq;
        double *o = node + k * FD_N_N;
        o[FD_N_RSDF] = rsdf;
        o[FD_N_INV_RSDF] = 1.0 / rsdf;
        *reinterpret_cast<float2 *>(o + FD_N_INV32) = make_float2(d2f_trunc(1.0 / rdq), d2f_trunc(1.0 / rsdf));
        const double is_s = 1.0 / (rsdf * rsdf), is_q = 1.0 / (rdq * rdq);
        const double a_sh = is_s + is_h, a_qh = is_q + is_h, a_sq = is_s + is_q;
        o[FD_N_A_SH] = a_sh;
        o[FD_N_I2A_SH] = 1.0 / (2.0 * a_sh);
        o[FD_N_A_QH] = a_qh;
        o[FD_N_I2A_QH] = 1.0 / (2.0 * a_qh);
        o[FD_N_A_SQ] = a_sq;
        o[FD_N_I2A_SQ] = 1.0 / (2.0 * a_sq);
    }
    /* fdsph3d coefficients (src/sphfd.c:5937-5972) for every cell */
    for (long long k = tid; k < (long long)(nz - 1) * (ny - 1); k += stride) {
        const int zc = (int)(k / (ny - 1)), yc = (int)(k % (ny - 1));
        const double rr[2] = {z0r - h * (double)zc, z0r - h * (double)(zc + 1)};
        const double sq[2] = {ysin[yc], ysin[yc + 1]};
        double *o = cell + k * FD_C_N;
        for (int ri = 0; ri < 2; ri++)
            for (int qi = 0; qi < 2; qi++) {
                const double dfs = df * sq[qi];
                const double a = 1.0 / hsq + (1.0 / dqsq + 1. / (dfs * dfs)) / (rr[ri] * rr[ri]);
                o[FD_C_DIAG(ri, qi)] = a;
                o[FD_C_I2A(ri, qi)] = 1.0 / (2.0 * a);
            }
        for (int r7 = 0; r7 < 2; r7++)
            for (int q7 = 0; q7 < 2; q7++)
                for (int ri = 0; ri < 2; ri++)
                    for (int qi = 0; qi < 2; qi++)
                        for (int sx = 0; sx < 2; sx++) {
                            const double gg = (r7 == ri) ? 1.0 : -1.0, nn = (q7 == qi) ? 1.0 : -1.0, mm = sx ? 1.0 : -1.0;
                            const double df2s7 = df * (df * sq[q7]);
                            const double kk = gg / hsq + (nn / dqsq + mm / (df2s7 * sq[qi])) / (rr[r7] * rr[ri]);
                            o[FD_C_PROW(r7, q7, ri, qi, sx)] = 2.0 * kk;
                        }
        for (int ri = 0; ri < 2; ri++)
            for (int qi = 0; qi < 2; qi++)
                for (int rj = 0; rj < 2; rj++)
                    for (int qj = 0; qj < 2; qj++)
                        for (int sx = 0; sx < 2; sx++) {
                            const double gg = (ri == rj) ? 1.0 : -1.0, nn = (qi == qj) ? 1.0 : -1.0, mm = sx ? 1.0 : -1.0;
                            const double df2si = dfsq * sq[qi];
                            const double kk = gg / hsq + (nn / dqsq + mm / (df2si * sq[qj])) / (rr[ri] * rr[rj]);
                            o[FD_C_PAIR(ri, qi, rj, qj, sx)] = 2.0 * kk;
                        }
    }
}

/* ---------------------------------------------------------------------------------------------- */
/* per-CTA state                                                                                   */

/* state of the current walk */
struct WalkShared {
    /* ready queues (one per face in a sweep graph; a face walk uses queue 0), the queue of points
     * resuming a search for an inherited stencil state, idle workers, finished nodes, parked points
     * and wait pairs */
    int nq;
    int qhead[6], qtail[6], qcap[6], qbase[6];
    int rqhead, rqtail, rqcap, idle, ndone, npark, nwait, nphi;
    int status;
    int headw[8];
    unsigned long long exitkey;
    long long rounds, deferred;
    unsigned long long st[5];
};

struct Shared {
    WalkShared w;
    int stat;                /* the station's status at the last csync */
    int wall[6], dflag[6];
    int radius, rad0, reverse, headpref;
    float carry_t0, carry_t4;
    /* current face of a face walk */
    int face, layer, ulo, uhi, vlo, vhi, nuf, n, n_pad;
    /* current sweep graph: on/off, face instances, points; per face, the 27-bit masks of the
     * neighbour offsets a node of that face reads, and of those in its inner plane */
    int graph, gok, ninst, single, nodefer;
    unsigned gfaces;
    long long gM;
    unsigned ctxm[6], innm[6];
    unsigned rel[6][27];     /* see relation_word */
    int lstride, imax;       /* layout of the sweep-graph tables (see GraphSmem) */
    /* statistics */
    long long faces, node_updates;
    int sweeps;
    int restart_wall[8];
    long long cyc[6];
    long long gsweeps;
};

/* ordering of a worker's global and shared stores before the counters that publish them */
__device__ __forceinline__ void wfence(const Shared &) { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

/* barrier after which every branch that depends on the station's status (sh.stat) is taken by all threads */
__device__ __forceinline__ void csync(Shared &sh)
{
    __syncthreads();
    if (threadIdx.x == 0) sh.stat = *const_cast<volatile int *>(&sh.w.status);
    __syncthreads();
}

/* face frame for a face number known only at run time */
__device__ __forceinline__ fdn_frame frame_of(int f)
{
    switch (f) {
    case 0: return fd_face_frame[0];
    case 1: return fd_face_frame[1];
    case 2: return fd_face_frame[2];
    case 3: return fd_face_frame[3];
    case 4: return fd_face_frame[4];
    default: return fd_face_frame[5];
    }
}

/* order-preserving 32-bit image of a float time (ties of -0 and +0 kept equal) */
__device__ __forceinline__ unsigned okey32(float f)
{
    unsigned b = __float_as_uint(f);
    if (b == 0x80000000u) b = 0u;
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

/* stencil evaluations by kind (3-D, new-edge, 2-D, new-face, 1-D): the warp's counts in its
 * shared area, passed by value (a pointer), so that no per-thread memory is involved */
struct Counters {
    unsigned long long *n;
};

__device__ __forceinline__ void count_eval(Counters cn, int kind) { atomicAdd(&cn.n[kind], 1ull); }

/* coordinate of node (x,y,z) along a grid axis, and a node placed from face coordinates: selects on
 * registers (arrays indexed by a run-time axis would live in per-thread local memory, whose L1 lines
 * this kernel's large shared-memory carve-out leaves little room for) */
__device__ __forceinline__ int coord(int axis, int x, int y, int z) { return axis == 0 ? x : axis == 1 ? y : z; }

__device__ __forceinline__ void place(const fdn_frame &fr, int u, int v, int n, int &x, int &y, int &z)
{
    x = fr.axis_u == 0 ? u : fr.axis_v == 0 ? v : n;
    y = fr.axis_u == 1 ? u : fr.axis_v == 1 ? v : n;
    z = fr.axis_u == 2 ? u : fr.axis_v == 2 ? v : n;
}

/* ---------------------------------------------------------------------------------------------- */
/* warp workers                                                                                    */
/*                                                                                                 */
/* A walk — one face, or a whole sweep as one graph — is a dependency graph whose ready nodes sit   */
/* in queues.  Every warp of the CTA is an independent worker: it claims up to 32 ready nodes of    */
/* one face direction, evaluates them (one lane per node for the per-node steps, the stencil       */
/* trials of all its nodes spread over the 32 lanes), commits them and queues the nodes they       */
/* complete.  Warps meet only at shared-memory counters, so the FP64 work of some warps hides the  */
/* memory and control latency of the others, and a node starts as soon as its own inputs are      */
/* final.                                                                                          */
/*                                                                                                 */
/* Queues: positions are taken with an atomic on the tail and written after; every entry starts as */
/* -1, so a worker that claimed a position not yet written waits for it (briefly: the writer is    */
/* between two instructions).  Stores of a node's time and of its queue entries are ordered by     */
/* __threadfence_block before the counters that publish them.  Every wait is bounded: a worker     */
/* idle for FD_WAIT_CYCLES without progress sets the station's status and all workers leave the   */
/* walk; all idle with nothing queued and nodes left is reported the same way.                    */

#define NB_PAD 19                    /* context row stride: the 32 rows fall on distinct banks */
#define FD_WAIT_CYCLES (4ll << 30)   /* about 2 s at the maximum SM clock */
#ifndef FD_WALK_CYCLES
#define FD_WALK_CYCLES (1ll << 37)   /* about 66 s: no walk of a real grid comes near it */
#endif
#define FD_QSPIN (1 << 22)           /* polls of an unwritten queue entry before giving up */
#define FD_KEYED 0x80000000u         /* counter word: the node's sort key is final */

#define FD_DESC_ROW(F)                                                                              \
    make_desc<F>(0), make_desc<F>(1), make_desc<F>(2), make_desc<F>(3), make_desc<F>(4), make_desc<F>(5), \
    make_desc<F>(6), make_desc<F>(7), make_desc<F>(8), make_desc<F>(9), make_desc<F>(10), make_desc<F>(11), \
    make_desc<F>(12), make_desc<F>(13), make_desc<F>(14), make_desc<F>(15), make_desc<F>(16), make_desc<F>(17), \
    make_desc<F>(18), make_desc<F>(19), make_desc<F>(20), make_desc<F>(21)
__constant__ TrialDesc c_desc[FDN_NFACE * FDN_NTRIAL] = {FD_DESC_ROW(0), FD_DESC_ROW(1), FD_DESC_ROW(2),
                                                         FD_DESC_ROW(3), FD_DESC_ROW(4), FD_DESC_ROW(5)};

/* shared by the CTA: the trial descriptors of all six faces */
struct CtaSmem {
    TrialDesc desc[FDN_NFACE][FDN_NTRIAL];
};
constexpr int kCtaSmemBytes = (int)((sizeof(CtaSmem) + 15) & ~(size_t)15);

/* the longest list: the 2-D and 1-D trials of 32 nodes */
constexpr int kItems = (TK_NF - TK_2D0 + FDN_NTRIAL - TK_1D0) * 32;

/* one warp's chunk of up to 32 nodes; slot = lane of the node */
struct WarpSmem {
    double res[32][FDN_NTRIAL];            /* trial values (2-D: after the causality selection) */
    float t[32][NB_PAD];                   /* 18-node time context */
    float s[32][NB_PAD];                   /* 18-node slowness context */
    float s0[32], s4[32];                  /* stencil state entering the 2-D block; before it, step lengths */
    int z[32], y[32];                      /* grid z and y of the node */
    unsigned short items[kItems];          /* (slot << 5 | trial) to evaluate, trial-major */
    unsigned long long cnt[6];             /* stencil evaluations by kind (5 used) */
};
static_assert(sizeof(WarpSmem) % 16 == 0, "keeps the dependency bytes after the warp areas aligned");
constexpr int kSmemBase = kCtaSmemBytes + FD_WARPS * (int)sizeof(WarpSmem);

template <class T>
__device__ __forceinline__ T vload(const T &x) { return *const_cast<const volatile T *>(&x); }

/* A value that other warps may be changing, as one lane sees it: what a warp branches on before a collective.  (Each
 * lane's own vload may give another value, and lanes that then go another way leave the collective's mask unmet.)
 * All 32 lanes call. */
template <class T>
__device__ __forceinline__ T vload_warp(const T &x) { return __shfl_sync(0xffffffffu, vload(x), 0); }

__device__ __forceinline__ void nb_off(int k, int &du, int &dv)
{
    /* k = 0..7 over the 3x3 block without its centre, row by row */
    const int c = k < 4 ? k : k + 1;
    du = c % 3 - 1;
    dv = c / 3 - 1;
}

/* bits of the neighbours of fill index i that lie inside the face rectangle */
__device__ __forceinline__ unsigned inrect_mask(int iu, int iv, int nuf, int nvf)
{
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        int du, dv;
        nb_off(k, du, dv);
        const int ju = iu + du, jv = iv + dv;
        if (ju >= 0 && ju < nuf && jv >= 0 && jv < nvf) m |= 1u << k;
    }
    return m;
}

/* Guards as bit tests.  A node's facts: bits 0-17, the context's times that are below 1e9; bits 18-21,
 * u > 0, u < nu-1, v > 0, v < nv-1; bits 22-25, u > ulo, u < uhi, v > vlo, v < vhi; bits 26-29, the own-plane
 * neighbours whose time is not zero, in the order of dir_index.  A trial's guards (first-contact gates
 * excluded) pass if the node has every fact the trial needs: one AND and one compare in place of up to
 * seven dependent shared-memory loads and branches per trial, and one code for all faces in place of six.
 * A chunk's loads and guards went from 14 to 5 thousand cycles at 3.9 nodes (27x20x21), from 22 to 9 at 29. */
constexpr int dir_index(int du, int dv) { return du == 1 ? 0 : du == -1 ? 1 : dv == 1 ? 2 : 3; }

template <int F>
constexpr unsigned guard_need(int K)
{
    const fdn_trial tr = fd_face_trials[F][K];
    unsigned m = (unsigned)tr.need << 18 | (unsigned)tr.inside << 22;
    for (int c = 0; c < tr.nchk; c++) {
        const fdn_node n = tr.chk[c];
        m |= ((tr.chk_nonzero >> c) & 1) ? 1u << (26 + dir_index(n.du, n.dv)) : 1u << nb_index(n);
    }
    return m;
}

/* what the code below takes for granted about the trial tables: the corner trials look at the quadrants
 * (+,+) (-,+) (+,-) (-,-), whose seven other cell nodes are their floor; a non-zero test is on an own-plane
 * neighbour; and only in-plane trials (2-D and 1-D) can be head waves (steps_as_assumed has the 1-D trials) */
constexpr bool trials_as_assumed()
{
    for (int f = 0; f < FDN_NFACE; f++)
        for (int k = 0; k < FDN_NTRIAL; k++) {
            const fdn_trial tr = fd_face_trials[f][k];
            for (int c = 0; c < tr.nchk; c++)
                if (((tr.chk_nonzero >> c) & 1) && (tr.chk[c].w != 0 || (tr.chk[c].du != 0) == (tr.chk[c].dv != 0))) return false;
            if (tr.kind == FDN_3D) {
                const int du = k & 1 ? -1 : 1, dv = k & 2 ? -1 : 1;
                unsigned cell = 0;
                for (int i = 0; i < 7; i++) {
                    if (tr.t[i].du != 0 && tr.t[i].du != du) return false;
                    if (tr.t[i].dv != 0 && tr.t[i].dv != dv) return false;
                    cell |= 1u << nb_index(tr.t[i]);
                }
                if (__builtin_popcount(cell) != 7 || (cell >> 4) & 1u) return false;
            }
            if (tr.head && !(k >= TK_2D0 && k < TK_NF) && !(k > TK_1D0)) return false;
        }
    return true;
}
static_assert(trials_as_assumed(), "trial tables");

/* per face: each trial's needed facts, and the head trials */
struct FaceGuards {
    unsigned need[FDN_NTRIAL];
    unsigned head;
};
template <int F>
constexpr FaceGuards make_guards()
{
    FaceGuards g{};
    for (int k = 0; k < FDN_NTRIAL; k++) {
        g.need[k] = guard_need<F>(k);
        if (fd_face_trials[F][k].head) g.head |= 1u << k;
    }
    return g;
}
__constant__ FaceGuards c_guards[FDN_NFACE] = {make_guards<0>(), make_guards<1>(), make_guards<2>(),
                                               make_guards<3>(), make_guards<4>(), make_guards<5>()};

/* a trial with floor fl cannot lower a running minimum that is at most g (any earlier value of the running
 * minimum, rounded up, is such a bound): its accepted value is >= fl, and its rejection value 1e11 is not
 * below g (99999997952 is the float below 1e11) */
__device__ __forceinline__ bool prunable(float fl, float g) { return fl >= g && g <= 99999997952.f; }

struct Rect {
    int u, v, nu, nv, ulo, uhi, vlo, vhi;
};

/* Guards, pruning and the trials to evaluate before the 2-D block: gm = trials whose guards pass
 * (first-contact gates excluded), em = corner and 1-D trials that can lower the minimum, and
 * new-edge trials when no corner can run (their gate is then decided by the initial value).
 * t: the context's times; below: its bits below 1e9. */
__device__ __forceinline__ void guards(int face, const float (&t)[NB_N], unsigned below, const Rect &r,
                                       unsigned &gm, unsigned &em)
{
    const FaceGuards &fg = c_guards[face];
    const float tp = t[NB_POINT];
    unsigned m = below;
    m |= (r.u > 0 ? 1u << 18 : 0u) | (r.u < r.nu - 1 ? 1u << 19 : 0u) | (r.v > 0 ? 1u << 20 : 0u)
         | (r.v < r.nv - 1 ? 1u << 21 : 0u);
    m |= (r.u > r.ulo ? 1u << 22 : 0u) | (r.u < r.uhi ? 1u << 23 : 0u) | (r.v > r.vlo ? 1u << 24 : 0u)
         | (r.v < r.vhi ? 1u << 25 : 0u);
    m |= (t[5] != 0.f ? 1u << 26 : 0u) | (t[3] != 0.f ? 1u << 27 : 0u) | (t[7] != 0.f ? 1u << 28 : 0u)
         | (t[1] != 0.f ? 1u << 29 : 0u);
    gm = 0;
#pragma unroll
    for (int K = 0; K < FDN_NTRIAL; K++)
        if ((fg.need[K] & ~m) == 0u) gm |= 1u << K;
    /* the rejection value 1e11 can only lower a minimum above it; 99999997952 is the float below 1e11 */
    const bool high = tp > 99999997952.f;
    unsigned can = 0;
#pragma unroll
    for (int K = TK_3D0; K < TK_NE0; K++) {
        const int eu = NB_POINT + (K & 1 ? -1 : 1), ev = NB_POINT + (K & 2 ? -3 : 3), euv = eu + ev - NB_POINT;
        const float fl = fmaxf(fmaxf(fmaxf(t[eu], t[ev]), fmaxf(t[euv], t[13])), fmaxf(fmaxf(t[eu + 9], t[ev + 9]), t[euv + 9]));
        if (fl < tp || high) can |= 1u << K;
    }
    const unsigned lower = (t[5] < tp ? 1u : 0u) | (t[3] < tp ? 2u : 0u) | (t[7] < tp ? 4u : 0u) | (t[1] < tp ? 8u : 0u);
    can |= (t[13] < tp ? 1u << TK_1D0 : 0u) | lower << (TK_1D0 + 1);
    em = gm & can;
    if (!(gm & 0xFu) && tp > 1.0e9f) em |= gm & 0xF0u;   /* their floors are looked at by ne_prune */
}

/* drop from em the new-edge trials whose floor shows that they cannot lower the minimum */
__device__ __forceinline__ unsigned ne_prune(const TrialDesc *dsc, const float *t18, unsigned em)
{
    for (unsigned b = em & 0xF0u; b; b &= b - 1) {
        const int K = __ffs(b) - 1;
        float fl = t18[dsc[K].slot[0]];
        for (int k = 1; k < 5; k++) fl = fmaxf(fl, t18[dsc[K].slot[k]]);
        if (prunable(fl, t18[NB_POINT])) em &= ~(1u << K);
    }
    return em;
}

/* append the items (lane, K) for the trials K of `of` whose bit is set in the lane's em, node by node */
__device__ __forceinline__ int push_items(unsigned short *items, int n, unsigned em, unsigned of, int lane)
{
    em &= of;
    const int mine = __popc(em);
    int end = mine;   /* items of the lanes up to this one */
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += x;
    }
    unsigned short *to = items + n + end - mine;
    for (; em; em &= em - 1) *to++ = (unsigned short)((lane << 5) | (__ffs(em) - 1));
    return n + __shfl_sync(0xffffffffu, end, 31);
}
constexpr unsigned k2d = 0xFFu << TK_2D0;
constexpr unsigned k1d = 0x1Fu << TK_1D0;

/* ---- evaluation of the queued items ----
 *
 * An FP64 instruction occupies its sub-partition for 64 cycles whatever the number of active lanes, so a
 * stencil evaluated by one lane holds it for its whole serial length: some 140 instructions for a corner, 85 for
 * a new-edge or a 2-D trial.  That is the right form for a warp full of items.  A chunk of a forward
 * sweep has one to five corners and rarely more than one of the others; there four lanes share an
 * item, each taking the products, divisions or sums that do not depend on one another, in the
 * reference's order within every sum: some 60 and 45 instructions for up to eight items (two such passes for
 * nine to sixteen corners cost as much as one of the other form). */
#define FD_QUAD 8

__device__ __forceinline__ double shfl_d(double x, int src) { return __shfl_sync(0xffffffffu, x, src); }

/* the accepted root of fdsphne / fdsph2d and of fdsph3d (tie rules of roots_2 and roots_3d) */
__device__ __forceinline__ double pick_2(double x1, double x2, double tmx)
{
    const bool bad1 = lt(x1, tmx), bad2 = lt(x2, tmx);
    return bad1 ? (bad2 ? 1.e11 : x2) : (bad2 ? x1 : (lt(x2, x1) ? x2 : x1));
}
__device__ __forceinline__ double pick_3(double x1, double x2, double tmx)
{
    const bool bad1 = lt(x1, tmx), bad2 = lt(x2, tmx);
    return bad1 ? (bad2 ? 1.e11 : x2) : (bad2 ? x1 : (lt(x1, x2) ? x1 : x2));
}

/* Up to eight corner items (fdsph3d, as eval_3d), lanes 4g .. 4g+3 on item g.  Lane r holds terms r and
 * r+4 of the seven; the pair sums' rows go 0 | 1 and 5 | 2 and 4 | 3 to the lanes, six products each; then lane
 * 0 adds up b, lane 1 c and lane 2 the slownesses, side by side.  Terms pass through the trial values'
 * columns from the 2-D trials on, which hold nothing yet: rows 4g .. 4g+3, T then R | S | P | Q.
 * Groups beyond n repeat the first item and store nothing. */
__device__ void eval_corners_quad(const fd_station_dev &sd, const TrialDesc *dsc, WarpSmem &ws, const unsigned short *items,
                                  int n, int lane)
{
    const int g = lane >> 2, r = lane & 3, lead = lane & ~3;
    const unsigned it = items[g < n ? g : 0];
    const int slot = (int)(it >> 5), K = (int)(it & 31);
    const TrialDesc &d = dsc[K];
    const float *t18 = ws.t[slot], *s18 = ws.s[slot];
    double *T = &ws.res[lead][TK_2D0], *R = T + 7, *S = &ws.res[lead + 1][TK_2D0], *P = &ws.res[lead + 2][TK_2D0],
           *Q = &ws.res[lead + 3][TK_2D0];
    int zc = ws.z[slot] + d.zmin, yc = ws.y[slot] + d.ymin;
    if (!FD_OK(zc, sd.g.nz - 1, 6) || !FD_OK(yc, sd.g.ny - 1, 7)) { zc = 0; yc = 0; }
    const double *C = sd.g.cell + (long long)(zc * (sd.g.ny - 1) + yc) * FD_C_N;
    const double a = C[d.a_idx], i2a = C[d.i2a_idx];
    float tm = 0.f;
    double tr = 0.0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = r + 4 * h;   /* term 7: the point itself, a slowness only */
        const int nb = i < 7 ? d.slot[i] : NB_POINT;
        S[i] = f2d(s18[nb]);
        if (i < 7) {
            const double t = f2d(t18[nb]);
            if (h == 0) tr = t;
            tm = h == 0 ? t18[nb] : fmaxf(tm, t18[nb]);
            T[i] = t;
            P[i] = t * C[d.prow[i]];
            Q[i] = (t * t) * C[d.diag[i]];
        }
    }
    tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 1));
    tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 2));
    __syncwarp();
    const int len = 6 - r, first = r == 0 ? 0 : r == 1 ? 6 : r == 2 ? 11 : 15;   /* row r's terms in the pair list */
    double acc = 0.0, acc2 = 0.0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const bool in = k < len;
        const double x = T[in ? r + 1 + k : k == 4 ? 5 : 6] * C[d.pair[in ? first + k : k + (r == 1 ? 15 : 14)]];
        if (k == 0) {
            acc = x;
        } else {
            const double y = (in ? acc : acc2) + x;
            if (in) acc = y;
            else acc2 = k == len ? x : y;
        }
    }
    const double r1 = acc * tr, r2 = acc2 * T[r == 1 ? 5 : 4];
    R[r] = r1;
    if (r == 1) R[5] = r2;
    if (r == 2) R[4] = r2;
    __syncwarp();
    const double *ch = r == 0 ? P : r == 1 ? Q : S;
    double v = ch[0];
#pragma unroll
    for (int k = 1; k < 7; k++) v = v + ch[k];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const double x = r == 1 ? R[k] : S[7];
        if (r == 1 || (r > 1 && k == 0)) v = v + x;
    }
    /* b*b in lane 0, 2 sum (sum / 8) in lane 2 */
    const double m = (r == 0 ? v : 2. * v) * (r == 0 ? v : 0.125 * v);
    const double b = shfl_d(v, lead), bb = shfl_d(m, lead);
    const double c = shfl_d(v, lead + 1) - shfl_d(m, lead + 2);
    const double rad = bb - 4. * a * c;
    const bool none = !(rad >= 0.);
    const double sq = __dsqrt_rn(none ? 0.0 : rad);
    const double x = div_rn(-b + (r & 1 ? -sq : sq), 2. * a, i2a);
    const double x1 = shfl_d(x, lead), x2 = shfl_d(x, lead + 1);
    if (r == 0 && g < n) ws.res[slot][K] = none ? 1.e11 : pick_3(x1, x2, f2d(tm));
    __syncwarp();
}

/* Up to eight new-edge or 2-D items (fdsphne and fdsph2d, as eval_ne and eval_2d), lanes 4g .. 4g+3 on item
 * g.  Both solve the same form, with X, Y, Z = t4, t2, t1 (new edge) or t1, t2, t3 (2-D):
 *   p = (X - Z)/dp - Y/dy,  q = (Y - Z)/dq - X/dx,  b = 2 (p/dy + q/dx),  c = p^2 + q^2 [+ ((t0 - t3)/d01)^2] - sum^2/4.
 * Lanes 0 to 3 take the four quotients, then 1 and 3 the two of b and 0 the new edge's third square. */
__device__ void eval_edges_quad(const fd_station_dev &sd, const TrialDesc *dsc, WarpSmem &ws, const unsigned short *items,
                                int n, int lane)
{
    const int g = lane >> 2, r = lane & 3, lead = lane & ~3;
    const unsigned it = items[g < n ? g : 0];
    const int slot = (int)(it >> 5), K = (int)(it & 31);
    const bool ne = K < TK_2D0;
    const TrialDesc &d = dsc[K];
    const float *t18 = ws.t[slot], *s18 = ws.s[slot];
    const int z = ws.z[slot], y = ws.y[slot];
    const int j = (ne ? 0x4132 : 0x0312) >> (4 * r) & 15;   /* this lane's distance: dp dy dq dx */
    double dd, iv, a, i2a;
    dist_rt(sd.g, d.dcls[j], z + d.ddz[j], y + d.ddy[j], dd, iv);
    apair_rt(sd.g, d.apair, z, y, a, i2a);
    const float fx = t18[d.slot[ne ? 4 : 1]], fy = t18[d.slot[2]], fz = t18[d.slot[ne ? 1 : 3]];
    float fl = fmaxf(fmaxf(fx, fy), fz);
    const double tz = f2d(fz), ta = f2d(r == 0 || r == 3 ? fx : fy);
    const double df = ta - tz;
    const double q1 = div_rn(r & 1 ? ta : df, dd, iv);
    const double pq = q1 - shfl_d(q1, lane ^ 1);      /* p in lane 0, q in lane 2 */
    double v = shfl_d(pq, lane & ~1);                 /* p in lanes 0 and 1, q in 2 and 3 */
    double d3 = 0.0;
    if (ne) {
        const float f0 = t18[d.slot[0]], f3 = t18[d.slot[3]];
        fl = fmaxf(fl, fmaxf(f0, f3));
        d3 = f2d(f0) - f2d(f3);
        if (r == 0) dist_rt(sd.g, d.dcls[0], z + d.ddz[0], y + d.ddy[0], dd, iv);
    } else {
        fl = fmaxf(fl, fmaxf(ws.s0[slot], ws.s4[slot]));
    }
    const double q2 = div_rn(r == 0 ? d3 : v, dd, iv);
    if (r == 0) v = q2;                               /* the new edge's third term; zero for a 2-D trial */
    const double b = 2. * (shfl_d(q2, lead + 1) + shfl_d(q2, lead + 3));
    /* slownesses in the reference's order, one conversion a lane */
    const int so = ne ? (r == 3 ? NB_POINT : d.slot[r == 0 ? 1 : r == 1 ? 2 : 4]) : (r == 0 ? NB_POINT : d.slot[r]);
    const double sl = f2d(s18[so]);
    const double sum = ((shfl_d(sl, lead) + shfl_d(sl, lead + 1)) + shfl_d(sl, lead + 2)) + shfl_d(sl, lead + 3);
    const double m = (r == 2 ? sum : v) * (r == 2 ? 0.25 * sum : v);
    const double c = ((shfl_d(m, lead + 1) + shfl_d(m, lead + 3)) + shfl_d(m, lead)) - shfl_d(m, lead + 2);
    const double rad = b * b - 4. * a * c;
    const bool none = !(rad >= 0.);
    const double sq = __dsqrt_rn(none ? 0.0 : rad);
    const double x = div_rn(-b + (r & 1 ? -sq : sq), 2. * a, i2a);
    const double x1 = shfl_d(x, lead), x2 = shfl_d(x, lead + 1);
    if (r == 0 && g < n) ws.res[slot][K] = none ? 1.e11 : pick_2(x1, x2, f2d(fl));
    __syncwarp();
}

/* Evaluate items[0..n), all corner trials (kind 0), new-edge (1), 2-D (2) or 1-D (4), with the warp's lanes; a
 * 2-D value is stored after the causality selection against its floor, which includes the stencil
 * state entering the 2-D block (src/sphfd.c:6116-6121).  Corners come in warps: whole warps of them, and a
 * remainder above FD_QUAD, take a lane each.  New-edge and 2-D items are rarely more than eight. */
template <int KIND>
__device__ __forceinline__ void eval_items(const fd_station_dev &sd, const TrialDesc *dsc, WarpSmem &ws,
                                           const unsigned short *items, int n, int lane)
{
    if (n == 0) return;
    if (lane == 0) ws.cnt[KIND] += (unsigned)n;
    if constexpr (KIND == 1 || KIND == 2) {
        for (int j0 = 0; j0 < n; j0 += 8) eval_edges_quad(sd, dsc, ws, items + j0, n - j0 < 8 ? n - j0 : 8, lane);
    } else {
        int j0 = 0;
        if constexpr (KIND == 0) {
            const int rest = n & 31;
            if (rest && rest <= FD_QUAD) {
                eval_corners_quad(sd, dsc, ws, items, rest, lane);
                j0 = rest;
            }
        }
        for (int j = j0 + lane; j < n; j += 32) {
            const unsigned it = items[j];
            const int slot = (int)(it >> 5), K = (int)(it & 31);
            const int z = ws.z[slot], y = ws.y[slot];
            if constexpr (KIND == 0) ws.res[slot][K] = eval_3d(dsc[K], ws.t[slot], ws.s[slot], sd.g, z, y);
            else ws.res[slot][K] = eval_1d(dsc[K], ws.t[slot], ws.s[slot], sd.g, z, y);
        }
    }
}

/* Replay of the corner and new-edge trials (every writer of the stencil state comes before the
 * 2-D block): the running minimum entering the 2-D block — an upper bound for every later trial's
 * turn — and the stale (t0,t4) the 2-D trials test against.  Returns em with the 2-D trials that can still
 * lower the minimum, and without the 1-D trials that cannot: nearly all lose to the corners by far more
 * than FP32 rounding, so their time is bounded from below in FP32 (step lengths truncated, products
 * rounded down and shortened by 2^-20, which covers the FP64 chain's rounding). */
__device__ unsigned stale_pair(const fd_station_dev &sd, const TrialDesc *dsc, WarpSmem &ws, int slot, int F,
                               unsigned gm, unsigned em, float it0, float it4)
{
    const float *t18 = ws.t[slot];
    const float dx = ws.s0[slot], dy = ws.s4[slot], dz = d2f_trunc(sd.g.h);   /* step lengths, put there with the context */
    double g1 = f2d(t18[NB_POINT]);
    float s0 = it0, s4 = it4;
    /* the last writer's slots are what remains of the writers before it */
    auto wrote = [&](unsigned writers) {
        const TrialDesc &d = dsc[31 - __clz((int)writers)];
        s0 = t18[d.slot[0]];
        s4 = t18[d.slot[4]];
    };
    auto lowest = [&](unsigned b) {
        for (; b; b &= b - 1) {
            const double v = ws.res[slot][__ffs(b) - 1];
            if (lt(v, g1)) g1 = v;
        }
    };
    if (gm & 0xFu) {
        wrote(gm & 0xFu);
        lowest(gm & em & 0xFu);
    }
    if ((gm & 0xF0u) && lt(1.0e9, g1)) {
        wrote(gm & 0xF0u);
        lowest(gm & em & 0xF0u);
    }
    ws.s0[slot] = s0;
    ws.s4[slot] = s4;
    const float gup = __double2float_ru(g1);
    *reinterpret_cast<float *>(&ws.res[slot][TK_NF]) = gup;   /* for filter_2d: the new-face value is never precomputed */
    unsigned add = 0;
    const float s04 = fmaxf(s0, s4);
    for (unsigned b = gm & k2d; b; b &= b - 1) {
        const int K = __ffs(b) - 1;
        const TrialDesc &d = dsc[K];
        const float fl = fmaxf(fmaxf(t18[d.slot[1]], t18[d.slot[2]]), fmaxf(t18[d.slot[3]], s04));
        if (!prunable(fl, gup)) add |= 1u << K;
    }
    if ((em & k1d) && gup <= 99999997952.f) {
        const fdn_frame fr = frame_of(F);
        const float *s18 = ws.s[slot];
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const int nb = k == 0 ? 13 : k == 1 ? 5 : k == 2 ? 3 : k == 3 ? 7 : 1;
            const int axis = k == 0 ? fr.axis_n : k < 3 ? fr.axis_u : fr.axis_v;
            const float len = axis == 0 ? dx : axis == 1 ? dy : dz;
            const float step = __fmul_rd(__fmul_rd(0.5f * (s18[NB_POINT] + s18[nb]), len), 0.99999904632568359375f);
            if (__fadd_rd(t18[nb], step) >= gup) em &= ~(1u << (TK_1D0 + k));
        }
    }
    return em | add;
}

/* Drop the queued 2-D items whose single-precision lower bound shows they cannot lower the
 * running minimum entering the 2-D block (kept in res[slot][TK_NF]); their value is recorded as the
 * rejection value, which leaves the minimum and the head-wave test as the true value would.
 * Compacts items[0..n) in place and returns the number left. */
__device__ int filter_2d(const fd_station_dev &sd, const TrialDesc *dsc, WarpSmem &ws, int n, int lane)
{
    int out = 0;
    for (int j0 = 0; j0 < n; j0 += 32) {
        const int j = j0 + lane;
        unsigned it = 0;
        bool keep = false;
        if (j < n) {
            it = ws.items[j];
            const int slot = (int)(it >> 5), K = (int)(it & 31);
            const TrialDesc &d = dsc[K];
            const float *t18 = ws.t[slot];
            const float fl = fmaxf(fmaxf(fmaxf(t18[d.slot[1]], t18[d.slot[2]]), fmaxf(t18[d.slot[3]], ws.s0[slot])),
                                   ws.s4[slot]);
            const float lo = lower_2d(d, t18, ws.s[slot], sd.g, ws.z[slot], ws.y[slot], fl);
            if (lo >= 0.f && prunable(lo, *reinterpret_cast<const float *>(&ws.res[slot][TK_NF])))
                ws.res[slot][K] = 1.e11;
            else
                keep = true;
        }
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if (keep) ws.items[out + __popc(b & ((1u << lane) - 1u))] = (unsigned short)it;
        out += __popc(b);
    }
    return out;
}

/* ---------------------------------------------------------------------------------------------- */
/* node addressing                                                                                 */

__device__ __forceinline__ unsigned long long node_key(float tin, int i)
{
    return ((unsigned long long)okey32(tin) << 32) | (unsigned)i;
}

/* grid extent and node strides of the time field and of the slowness model along an axis */
__device__ __forceinline__ int axis_len(const fd_station_dev &sd, int a) { return a == 0 ? sd.g.nx : a == 1 ? sd.g.ny : sd.g.nz; }
__device__ __forceinline__ long long t_stride(const fd_station_dev &sd, int a)
{
    return a == 0 ? 1ll : a == 1 ? (long long)sd.g.nx : (long long)sd.g.nx * sd.g.ny;
}
__device__ __forceinline__ long long s_stride(const fd_station_dev &sd, int a) { return a == 0 ? 1ll : a == 1 ? sd.s_sy : sd.s_sz; }

/* where a node sits: grid index, coordinates, face rectangle, fill index */
struct Where {
    long long p;
    int x, y, z;
    int i;       /* fill index in its face (instance) */
    int inst;    /* face instance of a sweep graph, -1 in a face walk */
    Rect r;
};

/* append e to a queue with tail counter `tail`; a position past the capacity (a node queued more
 * often than the walk allows) is refused */
__device__ __forceinline__ void enqueue_to(int *queue, int &tail, int cap, Shared &sh, int e)
{
    const int pos = atomicAdd(&tail, 1);
    if (pos < cap)
        *const_cast<volatile int *>(&queue[pos]) = e;   /* a strong store: readers synchronise on it */
    else
        atomicCAS(&sh.w.status, 0, 10);
}

/* ---------------------------------------------------------------------------------------------- */
/* face walks (one face at a time; used when the sweep-graph arrays are not available)             */

/* face walk: node i is final; mark it done and release its later in-face neighbours */
__device__ void face_release(const fd_station_dev &sd, Shared &sh, unsigned char *dag, int i, bool writer,
                             float st0, float st4)
{
    if (writer) {
        sd.scr.rec[i] = make_float2(st0, st4);
        atomicMax(&sh.w.exitkey, sd.scr.key[i]);
    } else {
        sd.scr.rec[i] = make_float2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
    }
    wfence(sh);
    /* done; a point waiting for the stencil state left before it resumes its search */
    const int waiter = atomicExch(&sd.scr.pst[i], -2);
    if (waiter >= 0) enqueue_to(sd.scr.rq, sh.w.rqtail, sh.w.rqcap, sh, waiter);
    const int nvf = sh.n / sh.nuf, iu = i % sh.nuf, iv = i / sh.nuf;
    const unsigned char *emask = dag + sh.n_pad;
    unsigned later = inrect_mask(iu, iv, sh.nuf, nvf) & ~(unsigned)emask[i];
    atomicOr(reinterpret_cast<unsigned *>(dag) + (i >> 2), 0xFFu << ((i & 3) * 8));
    while (later) {
        const int k = __ffs(later) - 1;
        later &= later - 1;
        int du, dv;
        nb_off(k, du, dv);
        const int j = (iv + dv) * sh.nuf + iu + du;
        const unsigned sh8 = (j & 3) * 8;
        const unsigned old = atomicSub(reinterpret_cast<unsigned *>(dag) + (j >> 2), 1u << sh8);
        if (((old >> sh8) & 0xFFu) == 1u) enqueue_to(sd.scr.queue, sh.w.qtail[0], sh.w.qcap[0], sh, j);
    }
}

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long x)
{
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
        x = y > x ? y : x;
    }
    return x;
}

/* ---------------------------------------------------------------------------------------------- */
/* sweep graphs                                                                                    */
/*                                                                                                 */
/* A whole sweep runs as one dependency graph.  Which face instance (a face at one wall position)  */
/* computes which node depends only on the walls, not on times, so the sweep's schedule of face    */
/* instances is simulated first; a node's owner then follows from two small shared-memory tables  */
/* (the instance of each face at each layer, and each instance's rectangle).  A node reads its     */
/* own-plane 3x3 block and the 3x3 block of its inner layer.  For each pair of nodes where one     */
/* reads the other and their owners differ, the earlier-owned one must finish first: the reader    */
/* needs its new value, or it must read the other's old one.  Within one face instance the order   */
/* is the sort order of the inner-layer times, known once a node's inner block is final (its inner */
/* block holds the inner nodes of all its in-face neighbours).  Every node keeps one counter word: */
/* inner block pending (bits 0-7), same-instance neighbours pending (8-15), other-instance nodes    */
/* pending (16-23), it made a writer call (bit 28), a point waits on it (bit 29), done (bit 30), key */
/* final (bit 31).  After a                                                                        */
/* restart (one face) this is a plane pipeline; in the forward sweep it lets all six faces and     */
/* successive wall positions advance together.                                                     */
/*                                                                                                 */
/* Inherited stencil state: a point whose 2-D trials need the state an earlier point left, and    */
/* whose result depends on it, waits for the last point before it (in the reference's order) that  */
/* made a writer call: the last such point in its own instance, once all keys there are final, or  */
/* the last one not yet done if that comes after it (then it looks again when that one is done),   */
/* else the last writer of the nearest earlier instance once that instance is complete.  Waits    */
/* are registered on a point (a wait pair and the counter's wait bit) or on an instance event (all */
/* keys final, all points done; a parked-point entry).                                            */

#ifndef FD_GRAPH_FORWARD
#define FD_GRAPH_FORWARD 1           /* the first sweep as a graph too */
#endif
#define FD_WRITERB 0x10000000u       /* done, and it made a writer call */
#define FD_WAITB 0x20000000u
#define FD_DONEB 0x40000000u

/* a face instance: face and layer, and its rectangle */
struct GRect {
    short fl, ulo, uhi, vlo, vhi, pad;
    __device__ __forceinline__ int face() const { return fl & 7; }
    __device__ __forceinline__ int layer() const { return fl >> 3; }
    __device__ __forceinline__ int nuf() const { return uhi - ulo + 1; }
};

/* In the dynamic shared memory after the warp areas (the face walks' dependency bytes otherwise).
 *
 * lay[a][c]: when the box's walls reach coordinate c of axis a, as an owner word (below): the instance
 * whose wall stands there, FD_IN_BOX if the sweep starts with c inside the box, FD_NEVER if no wall
 * gets there.  A node joins the box when the last of its three coordinates does, so its owner is the
 * largest of three entries: three shared-memory loads and two comparisons, where a search through the
 * six faces' instances and their rectangles took about a hundred instructions, divergent ones. */
#define FD_IN_BOX ((short)-1)
#define FD_NEVER ((short)0x7fff)
struct GraphSmem {
    short *lay[3];   /* entry c + 1 for coordinate c, FD_NEVER on both sides of the grid */
    GRect *rect;
    int *nkeyed, *ndone;   /* per instance: points whose sort key is final, points done */
};
static_assert((FD_IMAX << 3) + 7 < 0x7fff, "owner words in a short");

/* bytes of the tables for extents up to lmax and imax instances.  A launch asks for what its largest
 * station needs and no more: what shared memory leaves of the SM's 256 KB is L1, which the solver reads
 * its tables, times and keys through (28 KB beside the largest tables, 60 to 92 KB beside those of a
 * window; a 141x121x57 station 219 -> 177 ms). */
__host__ __device__ constexpr long long graph_smem_bytes(int lmax, int imax)
{
    return ((3ll * (lmax + 2) * 2 + 15) & ~15ll) + (long long)imax * (long long)(sizeof(GRect) + 2 * sizeof(int));
}

/* the tables of the largest grids, the warp areas and 2.5 KB of static shared memory fit a CTA's 227 KB */
static_assert(kSmemBase + graph_smem_bytes(FD_LMAX, FD_IMAX) + 2560 <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ GraphSmem gsmem(const Shared &sh)
{
    extern __shared__ __align__(16) unsigned char fd_dyn_smem[];
    short *l = reinterpret_cast<short *>(fd_dyn_smem + kSmemBase);
    const int n = sh.lstride;
    GRect *r = reinterpret_cast<GRect *>(fd_dyn_smem + kSmemBase + ((3 * n * 2 + 15) & ~15));
    int *c = reinterpret_cast<int *>(r + sh.imax);   /* GRect is 12 bytes */
    return {{l, l + n, l + 2 * n}, r, c, c + sh.imax};
}

/* Neighbour offsets (dx,dy,dz) are numbered k = (dz+1)*9 + (dy+1)*3 + (dx+1), 13 being the node
 * itself; the opposite offset is 26 - k.  An owner word holds (instance << 3) | face, -1 for a
 * node no instance of the sweep computes. */
__device__ __forceinline__ int own_inst(int w) { return w >> 3; }
__device__ __forceinline__ int own_face(int w) { return w & 7; }
__device__ __forceinline__ int owner_word(int lx, int ly, int lz)
{
    const int w = max(max(lx, ly), lz);
    return w == FD_NEVER ? -1 : w;
}

/* masks of the offsets a node of face f reads (own plane and inner plane) and of its inner plane */
__device__ void relation_masks(int f, unsigned &ctx, unsigned &inn)
{
    const fdn_frame fr = frame_of(f);
    ctx = 0;
    inn = 0;
    for (int k = 0; k < 27; k++) {
        if (k == 13) continue;
        const int on = coord(fr.axis_n, k % 3 - 1, (k / 3) % 3 - 1, k / 9 - 1);
        if (on == 0 || on == fr.inner) ctx |= 1u << k;
        if (on == fr.inner) inn |= 1u << k;
    }
}

/* What the node at offset k from a node of face F has to do with it.  Bits 0-5: it waits for that node
 * if it belongs to a later instance of face (bit) — it reads that node, or that node reads it; bits 6-11:
 * through its inner block; bit 12: k lies in F's plane, and then bits 16-19: its place in the inner 3x3
 * block relative to the centre, plus 4; bit 20: it comes later if the inner-layer times are equal. */
__device__ unsigned relation_word(const Shared &sh, int F, int k)
{
    unsigned w = 0;
    for (int f = 0; f < 6; f++) {
        if (((sh.ctxm[F] >> k) & 1u) || ((sh.ctxm[f] >> (26 - k)) & 1u)) w |= 1u << f;
        if ((sh.innm[f] >> (26 - k)) & 1u) w |= 1u << (6 + f);
    }
    const fdn_frame fr = frame_of(F);
    const int dx = k % 3 - 1, dy = (k / 3) % 3 - 1, dz = k / 9 - 1;
    if (coord(fr.axis_n, dx, dy, dz) == 0) {
        const int du = coord(fr.axis_u, dx, dy, dz), dv = coord(fr.axis_v, dx, dy, dz);
        w |= 1u << 12 | (unsigned)(dv * 3 + du + 4) << 16 | (dv > 0 || (dv == 0 && du > 0) ? 1u << 20 : 0u);
    }
    return w;
}

__device__ __forceinline__ int rect_n(const GRect &r) { return r.nuf() * (r.vhi - r.vlo + 1); }

/* owner word of node (x,y,z), which must lie in the grid */
__device__ __forceinline__ int owner_of(const GraphSmem &gs, int x, int y, int z)
{
    return owner_word(gs.lay[0][x + 1], gs.lay[1][y + 1], gs.lay[2][z + 1]);
}

/* a node's coordinates in one word: what the queues and lists of a sweep graph hold (extents are at most
 * FD_LMAX), so that nothing divides to get them back */
__device__ __forceinline__ int pack_xyz(int x, int y, int z) { return x | (y << 10) | (z << 20); }
static_assert(FD_LMAX <= 1024, "pack_xyz");
__device__ __forceinline__ int node_of(const fd_station_dev &sd, int xyz)
{
    return ((xyz >> 20) * sd.g.ny + ((xyz >> 10) & 1023)) * sd.g.nx + (xyz & 1023);
}

/* coordinates of point j of instance r, its node index */
__device__ __forceinline__ int inst_xyz(const GRect &r, int j)
{
    const int nuf = r.nuf(), iv = j / nuf;
    int x, y, z;
    place(frame_of(r.face()), r.ulo + j - iv * nuf, r.vlo + iv, r.layer(), x, y, z);
    return pack_xyz(x, y, z);
}
__device__ __forceinline__ int inst_node(const fd_station_dev &sd, const GRect &r, int j) { return node_of(sd, inst_xyz(r, j)); }

/* the in-face neighbour (du,dv) of a node comes later in its instance's order: inner-layer time (as
 * okey32 images), then fill index, which grows with dv and, within a row, with du */
__device__ __forceinline__ bool later_key(unsigned nb, unsigned own, int du, int dv)
{
    return nb > own || (nb == own && (dv > 0 || (dv == 0 && du > 0)));
}

/* Points parked on instance I's event `kind` (1: all keys final, 2: all done) go to the resume queue.  The
 * event's word heads a list of them through gpark, and says so once the event has fired; the one
 * thread whose count completes the event takes the list. */
FD_COLD void fire_event(const fd_station_dev &sd, Shared &sh, int I, int kind)
{
    wfence(sh);
    int k = atomicExch(&sd.scr.ginst[I].ev[kind - 1], FD_EV_FIRED);
    wfence(sh);
    while (k >= 0) {
        enqueue_to(sd.scr.grq, sh.w.rqtail, sh.w.rqcap, sh, vload(sd.scr.gpark[k].x));
        k = vload(sd.scr.gpark[k].y);
    }
}

/* Key event of a node (coordinates xyz, grid index q, instance I): its inner block is final, and its
 * later same-instance neighbours are dropped from its counter.  Returns the counter word after the
 * update. */
__device__ __forceinline__ unsigned key_event(const fd_station_dev &sd, Shared &sh, int I, int xyz, int q)
{
    const GraphSmem gs = gsmem(sh);
    const GRect r = gs.rect[I];
    const fdn_frame fr = frame_of(r.face());
    const int x = xyz & 1023, y = (xyz >> 10) & 1023, z = xyz >> 20;
    const int u = coord(fr.axis_u, x, y, z), v = coord(fr.axis_v, x, y, z);
    const int su = (int)t_stride(sd, fr.axis_u), sv = (int)t_stride(sd, fr.axis_v);
    const int qin = q + fr.inner * (int)t_stride(sd, fr.axis_n);   /* q's inner-layer node */
    /* columns and rows of the 3x3 block inside the rectangle */
    const unsigned in = (u > r.ulo ? 1u : 0u) | 2u | (u < r.uhi ? 4u : 0u) | (v > r.vlo ? 8u : 0u) | 16u | (v < r.vhi ? 32u : 0u);
    /* the inner-layer times of q and of its in-rectangle neighbours, all loads issued together */
    float tn[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const int du = k % 3 - 1, dv = k / 3 - 1;
        const unsigned bits = 1u << (du + 1) | 8u << (dv + 1);
        const int qk = qin + du * su + dv * sv;
        tn[k] = ((in & bits) == bits && FD_OK(qk, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 12)) ? sd.T[qk] : 0.f;
    }
    const unsigned kj = okey32(tn[4]);
    unsigned lat = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const int du = k % 3 - 1, dv = k / 3 - 1;
        const unsigned bits = 1u << (du + 1) | 8u << (dv + 1);
        if (k != 4 && (in & bits) == bits && later_key(okey32(tn[k]), kj, du, dv)) lat++;
    }
    if (!FD_OK(q, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 13) || !FD_OK(qin, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 29)
        || !FD_OK(I, sd.scr.ginst_cap, 14))
        return 0u;
    wfence(sh);
    const unsigned add = FD_KEYED - (lat << 8);
    const unsigned nw = atomicAdd(&sd.scr.gcnt[q], add) + add;
    if (!sh.nodefer && atomicAdd(&gs.nkeyed[I], 1) == rect_n(r) - 1) fire_event(sd, sh, I, 1);
    return nw;
}

__device__ __forceinline__ bool ready_word(unsigned w) { return (w & ~FD_WAITB) == FD_KEYED; }

__device__ __forceinline__ void graph_ready(const fd_station_dev &sd, Shared &sh, int face, int xyz)
{
    enqueue_to(sd.scr.gqueue + sh.w.qbase[face], sh.w.qtail[face], sh.w.qcap[face], sh, xyz);
}

/* Points that wait for a point: (awaited, waiting) pairs in a hash table probed one slot on at a time.  The
 * first word of a slot is -1 (free), -2 (being filled), -3 (taken back or woken) or the awaited point; a slot
 * never becomes free again within a sweep, so the pairs of a point lie between its hash slot and the
 * first free one.  (A list of all the sweep's pairs, searched for every awaited point, cost up to half a
 * million cycles a wake-up on windows with thousands of waits.) */
__device__ __forceinline__ unsigned wait_slot(int p) { return ((unsigned)p * 2654435761u) >> 15; }
static_assert(FD_GWAIT_CAP == 1 << 17, "wait_slot");

FD_COLD void wake_waiters(const fd_station_dev &sd, Shared &sh, int p)
{
    wfence(sh);
    unsigned k = wait_slot(p);
    for (int n = 0; n < FD_GWAIT_CAP; n++, k = (k + 1) & (FD_GWAIT_CAP - 1)) {
        const int x = vload(sd.scr.gwait[k].x);
        if (x == -1) break;
        if (x == p && atomicCAS(&sd.scr.gwait[k].x, p, -3) == p)
            enqueue_to(sd.scr.grq, sh.w.rqtail, sh.w.rqcap, sh, vload(sd.scr.gwait[k].y));
    }
}

/* node p (instance I, fill index i) is final: its record.  Returns its counter word as it was when it was
 * marked done: FD_WAITB if a point waits for it (the caller wakes those once it has used the time the
 * word takes to arrive).
 * The record and the exit key are both written before the done mark, but in no order between them: exit_floor, which reads
 * the key and then the record, may see a key without its record.  It only does so of a point that was open when
 * it read the flags, and then what it takes from the scan bounds that point's state, whatever the record holds (a NaN
 * falls out in its minimum); whoever reads a record as such has seen its done mark first. */
__device__ __forceinline__ unsigned graph_record(const fd_station_dev &sd, Shared &sh, long long p, int I, int i, bool writer,
                                                 float st0, float st4, float tin)
{
    if (!FD_OK(p, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 15) || !FD_OK(I, sd.scr.ginst_cap, 16)) return 0u;
    /* records: of every point when a point may need an earlier one's; else only the last instance's,
     * for the state the sweep leaves */
    if (!sh.nodefer || I == sh.ninst - 1) {
        if (writer) {
            sd.scr.grec[p] = make_float2(st0, st4);
            atomicMax(&sd.scr.ginst[I].exitkey, node_key(tin, i));
        } else {
            sd.scr.grec[p] = make_float2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
        }
    }
    wfence(sh);
    return sh.nodefer ? 0u : atomicOr(&sd.scr.gcnt[p], FD_DONEB | (writer ? FD_WRITERB : 0u));
}

/* nodes of a chunk up to which a release gives each neighbour a lane (more: each node), in a sweep of
 * several faces and of one */
#ifndef FD_FEW
#define FD_FEW 16
#endif
#ifndef FD_FEW1
#define FD_FEW1 6
#endif

/* a final node as its release needs it: packed coordinates, grid index, instance, its lane */
struct RelNode {
    int xyz, p, inst, slot;
};

/* what the node with owner word w at an offset with relation word rw drops from its counter when a
 * node of instance I is final (t13: that node's inner block centre) */
__device__ __forceinline__ unsigned release_dec(int w, int I, unsigned rw, const float *t13)
{
    const int oi = own_inst(w);
    if (w == FD_NEVER || oi < I) return 0u;
    if (oi == I) {
        /* a neighbour in the same instance waits only if it comes later */
        const unsigned a = okey32(t13[(int)((rw >> 16) & 15u) - 4]), b = okey32(*t13);
        return a > b || (a == b && (rw >> 20) & 1u) ? 1u << 8 : 0u;
    }
    const unsigned f = rw >> own_face(w);
    return !(f & 1u) ? 0u : (f & (1u << 6)) ? 1u : 1u << 16;
}

/* drop dec from the counter of node q (coordinates xyz); a node that becomes ready is queued, one whose
 * inner block is now complete goes on the list of key events */
__device__ __forceinline__ void release_one(const fd_station_dev &sd, Shared &sh, int q, int xyz, int fq, unsigned dec,
                                            int *keyq, int *nkey)
{
    if (!FD_OK(q, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 19)) return;
    const unsigned nw = atomicSub(&sd.scr.gcnt[q], dec) - dec;
    if (dec == 1u && (nw & 0xFFu) == 0u)
        keyq[atomicAdd(nkey, 1)] = xyz;
    else if (ready_word(nw))
        graph_ready(sd, sh, fq, xyz);
}

/* Release what waits on the chunk's final nodes (fin, was, wh: this lane's node, graph_record's word).  All 32
 * lanes call.
 *
 * What bounds a release is instructions: a warp of this kernel issues one about every ten cycles, so
 * what matters is how many the warp steps through.  A chunk of a forward sweep holds two to nine nodes;
 * each node's 26 neighbours then go to 26 lanes, so that a node costs one pass, and what depends on the
 * neighbour's offset alone (its relation word, its index offset) is set up once per chunk.  With more
 * nodes each lane walks the neighbours of its own node, with the offsets known at compile time (in a
 * one-face sweep only the 9 nodes of the next instance and the 8 of its own).  Nodes whose inner block
 * the chunk completes are collected (in the trial values' area, free after the commit) and take their
 * keys together: a key event is three more round trips to memory.
 *
 * Measured, commit and release of one chunk: 55 -> 28 thousand cycles at 3.8 nodes (27x20x21), 80 -> 50 at
 * 29 nodes (141x121x57), against a loop over the neighbours with a search of the six faces for each
 * owner and a key event inside it.  The two forms cost the same at about 16 nodes of a forward sweep (27
 * steps of the second form; 27x20x21 takes 2.5 % longer with the line at 8, 0.7 % at 12) and at 6 of a one-face
 * sweep (17 steps; 4 and 10 measure the same). */
__device__ void graph_release(const fd_station_dev &sd, Shared &sh, WarpSmem &ws, int F, bool fin, unsigned was,
                              const Where &wh)
{
    const int lane = threadIdx.x & 31;
    const GraphSmem gs = gsmem(sh);
    const unsigned mask = __ballot_sync(0xffffffffu, fin);
    const int m = __popc(mask);
    if (!m) return;
    static_assert(26 * 32 * sizeof(int) <= sizeof ws.res, "a node takes its key once, after one of at most 26 x 32 releases");
    int *keyq = reinterpret_cast<int *>(&ws.res[0][0]);
    int *nkey = reinterpret_cast<int *>(&ws.cnt[5]);
    const int nx = sd.g.nx, ny = sd.g.ny;
    const bool few = m <= (sh.single ? FD_FEW1 : FD_FEW);
    static_assert(FD_FEW <= 32 && FD_FEW1 <= 32 && 32 * sizeof(RelNode) <= sizeof ws.s0 + sizeof ws.s4 + sizeof ws.z + sizeof ws.y, "RelNode");
    RelNode *rn = reinterpret_cast<RelNode *>(ws.s0);   /* s0, s4, z, y: free after the commit */
    if (few && fin)
        rn[__popc(mask & ((1u << lane) - 1u))] = {pack_xyz(wh.x, wh.y, wh.z), (int)wh.p, wh.inst, lane};
    if (lane == 0) *nkey = 0;
    __syncwarp();
    wfence(sh);
    if (few) {
        if (lane < 26) {
            const int k = lane + (lane >= 13);
            const int kx = k % 3, ky = (k / 3) % 3, kz = k / 9;
            const int off = ((kz - 1) * ny + ky - 1) * nx + kx - 1, oxyz = kx - 1 + (ky - 1) * 1024 + (kz - 1) * (1 << 20);
            const unsigned rw = sh.rel[F][k];
            for (int j = 0; j < m; j++) {
                const RelNode n = rn[j];
                const int w = max(max(gs.lay[0][(n.xyz & 1023) + kx], gs.lay[1][((n.xyz >> 10) & 1023) + ky]),
                                  gs.lay[2][(n.xyz >> 20) + kz]);
                const unsigned dec = release_dec(w, n.inst, rw, &ws.t[n.slot][13]);
                if (dec) release_one(sd, sh, n.p + off, n.xyz + oxyz, own_face(w), dec, keyq, nkey);
            }
        }
    } else if (sh.single) {
        if (fin) {
            const fdn_frame fr = frame_of(F);
            const GRect r = gs.rect[wh.inst];
            const int su = (int)t_stride(sd, fr.axis_u), sv = (int)t_stride(sd, fr.axis_v);
            const int p = (int)wh.p, pn = p - fr.inner * (int)t_stride(sd, fr.axis_n);
            const int hu = 1 << (10 * fr.axis_u), hv = 1 << (10 * fr.axis_v);   /* steps of packed coordinates */
            const int xyz = pack_xyz(wh.x, wh.y, wh.z), xyzn = xyz - fr.inner * (1 << (10 * fr.axis_n));
            const float *t13 = &ws.t[lane][13];
            const unsigned own = okey32(*t13);
            /* columns (bits 0-2) and rows (3-5) of the 3x3 block inside a rectangle */
            auto inside = [&](const GRect &q) {
                const int u = wh.r.u, v = wh.r.v;
                return (u - 1 >= q.ulo && u - 1 <= q.uhi ? 1u : 0u) | (u >= q.ulo && u <= q.uhi ? 2u : 0u)
                       | (u + 1 >= q.ulo && u + 1 <= q.uhi ? 4u : 0u) | (v - 1 >= q.vlo && v - 1 <= q.vhi ? 8u : 0u)
                       | (v >= q.vlo && v <= q.vhi ? 16u : 0u) | (v + 1 >= q.vlo && v + 1 <= q.vhi ? 32u : 0u);
            };
            const unsigned mine = inside(r);
            const bool adj = wh.inst + 1 < sh.ninst && gs.rect[wh.inst + 1].layer() == r.layer() - fr.inner;
            const unsigned next = adj ? inside(gs.rect[wh.inst + 1]) : 0u;
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const int du = k % 3 - 1, dv = k / 3 - 1;
                const unsigned bits = 1u << (du + 1) | 8u << (dv + 1);
                const int o = du * su + dv * sv, oh = du * hu + dv * hv;
                if ((next & bits) == bits) release_one(sd, sh, pn + o, xyzn + oh, F, 1u, keyq, nkey);
                if (k != 4 && (mine & bits) == bits && later_key(okey32(t13[dv * 3 + du]), own, du, dv))
                    release_one(sd, sh, p + o, xyz + oh, F, 1u << 8, keyq, nkey);
            }
        }
    } else {
        if (fin) {
            /* (a loop, not 26 copies: the solver's code is larger than the instruction caches, and the copies
             * cost the sweeps that never get here more than the loop costs this one) */
            const int xyz = pack_xyz(wh.x, wh.y, wh.z), nxy = nx * ny;
            const float *t13 = &ws.t[lane][13];
            const short *ax = gs.lay[0] + wh.x, *ay = gs.lay[1] + wh.y, *az = gs.lay[2] + wh.z;
            int kx = 0, ky = 0, kz = 0, q = (int)wh.p - nxy - nx - 1, o = -(1 << 20) - 1024 - 1;
#pragma unroll 1
            for (int k = 0; k < 27; k++) {
                const int w = max(max(ax[kx], ay[ky]), az[kz]);
                const unsigned dec = k == 13 ? 0u : release_dec(w, wh.inst, sh.rel[F][k], t13);
                if (dec) release_one(sd, sh, q, xyz + o, own_face(w), dec, keyq, nkey);
                q++;
                o++;
                if (++kx == 3) {
                    kx = 0;
                    q += nx - 3;
                    o += 1024 - 3;
                    if (++ky == 3) {
                        ky = 0;
                        kz++;
                        q += nxy - 3 * nx;
                        o += (1 << 20) - 3 * 1024;
                    }
                }
            }
        }
    }
    __syncwarp();
    wfence(sh);
    if (was & FD_WAITB) wake_waiters(sd, sh, (int)wh.p);
    /* inner blocks now complete: these nodes' keys and in-face order are known */
    const int nk = *nkey;
    for (int j = lane; j < nk; j += 32) {
        const int q = keyq[j];
        const int w = owner_of(gs, q & 1023, (q >> 10) & 1023, q >> 20);
        if (ready_word(key_event(sd, sh, own_inst(w), q, node_of(sd, q)))) graph_ready(sd, sh, own_face(w), q);
    }
    __syncwarp();
}

/* point w waits for an event of instance I (kind 1: all keys final, 2: all points done) (lane 0) */
FD_COLD void wait_event(const fd_station_dev &sd, Shared &sh, int w, int I, int kind)
{
    const int k = atomicAdd(&sh.w.npark, 1);
    if (k >= FD_GPARK_CAP) {
        atomicCAS(&sh.w.status, 0, 15);
        return;
    }
    int *head = &sd.scr.ginst[I].ev[kind - 1];
    sd.scr.gpark[k].x = w;
    for (int h = vload(*head);;) {
        if (h == FD_EV_FIRED) {   /* it has happened already */
            enqueue_to(sd.scr.grq, sh.w.rqtail, sh.w.rqcap, sh, w);
            return;
        }
        sd.scr.gpark[k].y = h;
        wfence(sh);
        const int old = atomicCAS(head, h, k);
        if (old == h) return;
        h = old;
    }
}

/* point w waits for point p to be done (lane 0).  Returns false if p is already done (no wait). */
FD_COLD bool wait_point(const fd_station_dev &sd, Shared &sh, int w, long long p)
{
    if (atomicAdd(&sh.w.nwait, 1) >= FD_GWAIT_CAP) {
        atomicCAS(&sh.w.status, 0, 15);
        return true;
    }
    unsigned k = wait_slot((int)p);
    for (int n = 0; n < FD_GWAIT_CAP; n++, k = (k + 1) & (FD_GWAIT_CAP - 1))
        if (vload(sd.scr.gwait[k].x) == -1 && atomicCAS(&sd.scr.gwait[k].x, -1, -2) == -1) break;
    sd.scr.gwait[k].y = w;
    wfence(sh);
    atomicExch(&sd.scr.gwait[k].x, (int)p);
    wfence(sh);
    if (!(atomicOr(&sd.scr.gcnt[p], FD_WAITB) & FD_DONEB)) return true;
    /* p finished meanwhile: take the pair back unless p's release already took it (and queued w) */
    return atomicCAS(&sd.scr.gwait[k].x, (int)p, -3) != (int)p;
}

/* ---------------------------------------------------------------------------------------------- */
/* evaluation of one chunk                                                                         */

/* the head-wave measure of trial d against its threshold, as the reference forms it */
FD_COLD bool head_wave_exact(const fd_station_dev &sd, const TrialDesc &d, const float *s18, int z, int y, double num)
{
    return num / head_den(d, s18, sd.g, z, y) > FD_HEADTEST;
}

/* num / (length * slowness) > FD_HEADTEST for num >= 0.  Almost every quotient is far from the threshold: in
 * FP32 (num and the reciprocal length truncated, each within 2^-23) it tells unless the quotient is within
 * 2^-18 of it, and only then is the reference's product and division made (20 FP64 instructions). */
__device__ __forceinline__ bool head_wave(const fd_station_dev &sd, const TrialDesc &d, const float *s18, int z, int y,
                                          double num)
{
    const float2 f = inv32_at(sd.g, z + d.ddz[0], y + d.ddy[0]);
    const float iv = d.dcls[0] == CH_H ? d2f_trunc(sd.g.inv_h) : d.dcls[0] == CH_RDQ ? f.x : f.y;
    const float n = d2f_trunc(num) * iv, t = 1.e-3f * s18[NB_POINT];
    if (n > t * 1.0000038146972656f) return true;
    if (n < t * 0.9999961853027344f) return false;
    return head_wave_exact(sd, d, s18, z, y, num);
}

/* a new-edge or new-face value that was not computed with the chunk's items */
FD_COLD double contact_value(const fd_station_dev &sd, const TrialDesc &d, const float *t18, const float *s18, int z, int y,
                             bool nf)
{
    return nf ? eval_nf(d, t18, s18, sd.g, z, y) : eval_ne(d, t18, s18, sd.g, z, y);
}

/* The reference's sequential minimum over the 22 trials of one node, from the values computed
 * by the warp (new-edge and new-face values that were not precomputed are evaluated here — they
 * are needed only at first contact), then the commit (src/sphfd.c:1756-1760) and the node's
 * stencil-state record; a face walk also releases the nodes that wait on it here.
 *
 * `permissive`: the node makes no writer call before its 2-D trials, so those test against a
 * stencil state left by an earlier point; their values were computed with no stale floor.  A
 * stale floor can only turn a 2-D value into the rejection value, so if no 2-D value lowered
 * the running minimum the result is the one the true state gives and the node commits; else it
 * returns false without committing. */
__device__ bool commit_node(const fd_station_dev &sd, Shared &sh, const TrialDesc *dsc, WarpSmem &ws, int slot,
                            int F, const Where &wh, unsigned gm, unsigned em, float it0, float it4, bool permissive,
                            unsigned char *dag, unsigned &was, Counters cn)
{
    const float *t18 = ws.t[slot], *s18 = ws.s[slot];
    const double told = f2d(t18[NB_POINT]);
    const int z = ws.z[slot], y = ws.y[slot];
    double guess = told;
    const unsigned head = c_guards[F].head;
    int lastK = -1, writer = -1;   /* the last head trial that lowered the minimum; the last writer */
    double last_gb = 0.0, last_v = 0.0;
    auto take = [&](int K, double v) {
        if (!lt(v, guess)) return false;
        if ((head >> K) & 1u) { lastK = K; last_gb = guess; last_v = v; }
        guess = v;
        return true;
    };
    /* new-edge and new-face trials run only while the minimum is above 1e9, tested on entry to their
     * block (src/sphfd.c:1375, :1698); a value not precomputed is evaluated unless it cannot improve */
    auto contact = [&](int K) {
        const TrialDesc &d = dsc[K];
        writer = K;
        if ((em >> K) & 1u) {
            take(K, ws.res[slot][K]);
            return;
        }
        float fl = t18[d.slot[0]];
        for (int k = 1; k < 5; k++) fl = fmaxf(fl, t18[d.slot[k]]);
        if (prunable(fl, __double2float_ru(guess))) return;
        take(K, contact_value(sd, d, t18, s18, z, y, K == TK_NF));
        count_eval(cn, K == TK_NF ? 3 : 1);
    };
    if (gm & 0xFu) writer = 31 - __clz((int)(gm & 0xFu));
    for (unsigned b = gm & em & 0xFu; b; b &= b - 1) take(__ffs(b) - 1, ws.res[slot][__ffs(b) - 1]);
    if ((gm & 0xF0u) && lt(1.0e9, guess))
        for (unsigned b = gm & 0xF0u; b; b &= b - 1) contact(__ffs(b) - 1);
    bool win2d = false;
    for (unsigned b = gm & em & k2d; b; b &= b - 1) win2d |= take(__ffs(b) - 1, ws.res[slot][__ffs(b) - 1]);
    if (((gm >> TK_NF) & 1u) && lt(1.0e9, guess)) contact(TK_NF);
    for (unsigned b = gm & em & (0x1Fu << TK_1D0); b; b &= b - 1) take(__ffs(b) - 1, ws.res[slot][__ffs(b) - 1]);
    if (permissive && win2d) return false;
    if (lt(guess, told) && FD_OK(wh.p, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 11)) {
        sd.T[wh.p] = __double2float_rn(guess);
        if (lastK >= 0) {
            /* only the last head trial that lowered the minimum sets the measure that is tested */
            if (head_wave(sd, dsc[lastK], s18, z, y, last_gb - last_v)) atomicAdd(&sh.w.headw[frame_of(F).headw], 1);
        }
    }
    const float st0 = writer < 0 ? it0 : t18[dsc[writer].slot[0]], st4 = writer < 0 ? it4 : t18[dsc[writer].slot[4]];
    if (sh.graph)
        was = graph_record(sd, sh, wh.p, wh.inst, wh.i, writer >= 0, st0, st4, t18[13]);
    else
        face_release(sd, sh, dag, wh.i, writer >= 0, st0, st4);
    return true;
}

/* where the node of queue entry e lies: a fill index in a face walk, packed coordinates in a graph;
 * ok false for a graph node no instance owns */
__device__ __forceinline__ Where locate(const fd_station_dev &sd, const Shared &sh, int F, int e, bool &ok)
{
    const fdn_frame fr = frame_of(F);
    Where wh;
    ok = true;
    if (sh.graph) {
        wh.p = node_of(sd, e);
        wh.x = e & 1023;
        wh.y = (e >> 10) & 1023;
        wh.z = e >> 20;
        const int w = owner_of(gsmem(sh), wh.x, wh.y, wh.z);
        if (w < 0) {
            ok = false;
            return wh;
        }
        wh.inst = own_inst(w);
        const GRect gr = gsmem(sh).rect[wh.inst];
        wh.r.u = coord(fr.axis_u, wh.x, wh.y, wh.z);
        wh.r.v = coord(fr.axis_v, wh.x, wh.y, wh.z);
        wh.r.ulo = gr.ulo; wh.r.uhi = gr.uhi; wh.r.vlo = gr.vlo; wh.r.vhi = gr.vhi;
        wh.i = (wh.r.v - gr.vlo) * gr.nuf() + wh.r.u - gr.ulo;
    } else {
        wh.i = e;
        wh.inst = -1;
        wh.r.u = sh.ulo + e % sh.nuf;
        wh.r.v = sh.vlo + e / sh.nuf;
        wh.r.ulo = sh.ulo; wh.r.uhi = sh.uhi; wh.r.vlo = sh.vlo; wh.r.vhi = sh.vhi;
        place(fr, wh.r.u, wh.r.v, sh.layer, wh.x, wh.y, wh.z);
        wh.p = ((long long)wh.z * sd.g.ny + wh.y) * sd.g.nx + wh.x;
    }
    wh.r.nu = axis_len(sd, fr.axis_u);
    wh.r.nv = axis_len(sd, fr.axis_v);
    return wh;
}

/* Queue a point whose 2-D trials (which) won without the state it inherits.  Its record, not read while it is pending,
 * takes the lowest of their values: what that state must exceed to reject them all (exit_floor). */
FD_COLD void defer(const fd_station_dev &sd, Shared &sh, const WarpSmem &ws, int slot, long long p, unsigned which, int e)
{
    if (sh.graph) {
        double low = 1.e11;
        for (; which; which &= which - 1) {
            const double v = ws.res[slot][__ffs(which) - 1];
            if (lt(v, low)) low = v;
        }
        sd.scr.grec[p].x = __double2float_ru(low);
        wfence(sh);
    }
    enqueue_to(sh.graph ? sd.scr.grq : sd.scr.rq, sh.w.rqtail, sh.w.rqcap, sh, e);
}

/* a float from global to shared memory without a register (waited for with cp.async.wait_all): the
 * slownesses are first needed by the trials, after the guards that the times alone decide */
__device__ __forceinline__ void copy_async4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

/* Evaluate and commit one chunk of face F: lane l holds queue entry e (-1 for none).  A node given
 * with inherit kState uses (it0, it4) as the stencil state entering it; with kFloor it0 is a floor of that
 * state's larger time, and the node commits if no 2-D trial wins above it.  All 32 lanes call. */
enum { kNoState, kState, kFloor };
__device__ void warp_chunk(const fd_station_dev &sd, Shared &sh, const CtaSmem &cs, WarpSmem &ws, int F, int e,
                           int inherit, float it0, float it4, unsigned char *dag, Counters cn)
{
    const int lane = threadIdx.x & 31;
    const fdn_frame fr = frame_of(F);
    const TrialDesc *dsc = cs.desc[F];
    Where wh;
    unsigned gm = 0, em = 0;
    bool permissive = false;
    FD_TIC(ta);
    if (e >= 0) {
        bool ok;
        wh = locate(sd, sh, F, e, ok);
        if (!ok) {
            atomicCAS(&sh.w.status, 0, 14);   /* a queued node no face instance owns */
            e = -1;
        }
    }
    const bool valid = e >= 0;
    if (valid) {
        const float *pT = sd.T + wh.p;
        const float *pS = sd.S + ((long long)wh.z * sd.s_sz + (long long)wh.y * sd.s_sy + wh.x);
        ws.z[lane] = wh.z;
        ws.y[lane] = wh.y;
        float *tr = ws.t[lane], *sr = ws.s[lane];
        const int su = (int)t_stride(sd, fr.axis_u), sv = (int)t_stride(sd, fr.axis_v);
        const long long ssu = s_stride(sd, fr.axis_u), ssv = s_stride(sd, fr.axis_v);
        const int inner_t = fr.inner * (int)t_stride(sd, fr.axis_n);   /* a plane has at most 2^30 nodes */
        const long long inner_s = fr.inner * s_stride(sd, fr.axis_n);
        /* columns (bits 0-2) and rows (bits 3-5) of the block inside the grid */
        const unsigned inside = (wh.r.u > 0 ? 1u : 0u) | 2u | (wh.r.u < wh.r.nu - 1 ? 4u : 0u) | (wh.r.v > 0 ? 8u : 0u)
                                | 16u | (wh.r.v < wh.r.nv - 1 ? 32u : 0u);
        float t[NB_N];
#pragma unroll
        for (int nb = 0; nb < NB_N; nb++) {
            const int w = nb / 9, dv = (nb / 3) % 3 - 1, du = nb % 3 - 1;
            const unsigned bits = 1u << (du + 1) | 8u << (dv + 1);
            t[nb] = 0.f;
            if ((inside & bits) == bits) {
                const int o = du * su + dv * sv + (w ? inner_t : 0);
                if (FD_OK(wh.p + o, (long long)sd.g.nx * sd.g.ny * sd.g.nz, 27)) {
                    t[nb] = pT[o];   /* the CTA's own stores keep its L1 current */
                    copy_async4(&sr[nb], pS + (du * ssu + dv * ssv + (w ? inner_s : 0ll)));
                }
            } else {
                sr[nb] = 0.f;
            }
        }
        unsigned below = 0;
#pragma unroll
        for (int nb = 0; nb < NB_N; nb++) {
            tr[nb] = t[nb];
            if (t[nb] < 1.e9f) below |= 1u << nb;
        }
        guards(F, t, below, wh.r, gm, em);
        /* the point's step lengths along x and y for the 1-D bounds (see stale_pair) */
        ws.s0[lane] = d2f_trunc(node_row(sd.g, wh.z, wh.y)[FD_N_RSDF]);
        ws.s4[lane] = d2f_trunc(sd.g.zrow[(long long)(FD_OK(wh.z, sd.g.nz, 8) ? wh.z : 0) * FD_Z_N + FD_Z_RDQ]);
        if (em & 0xF0u) em = ne_prune(dsc, tr, em);
        /* a 2-D trial before any corner / new-edge call reads the state an earlier point left */
        permissive = inherit != kState && (gm & 0xFu) == 0 && !((gm & 0xF0u) && t[NB_POINT] > 1.0e9f) && (gm & 0xFF00u);
    }
    __syncwarp();
    const int n3 = push_items(ws.items, 0, em, 0xFu, lane);
    const int n1 = push_items(ws.items, n3, em, 0xF0u, lane);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    FD_TOC(1, ta);
    FD_TIC(tb);
    eval_items<0>(sd, dsc, ws, ws.items, n3, lane);
    eval_items<1>(sd, dsc, ws, ws.items + n3, n1 - n3, lane);
    __syncwarp();
    const float lo = inherit == kFloor ? it0 : __int_as_float(0xff800000);   /* -inf: no stale floor */
    const float p0 = permissive ? lo : it0, p4 = permissive ? lo : it4;
    if (valid) em = stale_pair(sd, dsc, ws, lane, F, gm, em, p0, p4);
    __syncwarp();
    int n2 = push_items(ws.items, 0, em, k2d, lane);
    __syncwarp();
    n2 = filter_2d(sd, dsc, ws, n2, lane);
    const int n4 = push_items(ws.items, n2, em, k1d, lane);
    __syncwarp();
    eval_items<2>(sd, dsc, ws, ws.items, n2, lane);
    eval_items<4>(sd, dsc, ws, ws.items + n2, n4 - n2, lane);
    __syncwarp();
    FD_TOC(2, tb);
    FD_TIC(tc);
    bool fin = false;
    unsigned was = 0;   /* graph_record's word */
    if (valid) {
        fin = commit_node(sd, sh, dsc, ws, lane, F, wh, gm, em, p0, p4, permissive, dag, was, cn);
        if (!fin) {
            if (inherit != kFloor) atomicAdd(reinterpret_cast<unsigned long long *>(&sh.w.deferred), 1ull);
            if (sh.nodefer)
                atomicCAS(&sh.w.status, 0, 6);   /* excluded by the sweep's precondition */
            else
                defer(sd, sh, ws, lane, wh.p, gm & em & k2d, e);
        }
    }
    if (sh.graph) graph_release(sd, sh, ws, F, fin, was, wh);
    if (sh.graph && !sh.nodefer) {
        /* points done per face instance, one atomic per instance in the chunk; the instance
         * complete wakes points waiting for its last writer */
        const int key = fin ? wh.inst : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        if (fin && lane == __ffs(peers) - 1) {
            const int c = __popc(peers);
            const int old = atomicAdd(&gsmem(sh).ndone[key], c);
            if (old + c == rect_n(gsmem(sh).rect[key])) fire_event(sd, sh, key, 2);
        }
    }
    const unsigned done = __ballot_sync(0xffffffffu, fin);
    if (lane == 0 && done) {
        wfence(sh);
        atomicAdd(&sh.w.ndone, __popc(done));
    }
    __syncwarp();
    FD_TOC(3, tc);
}

/* ---------------------------------------------------------------------------------------------- */
/* inherited stencil state                                                                         */

/* face walk: the point that precedes point c in sort order (largest key below c's), -1 if none */
__device__ int predecessor(const fd_station_dev &sd, int n, int c, int lane)
{
    const unsigned long long kc = sd.scr.key[c];
    unsigned long long best = 0ull;   /* every key is above 0: times are not negative */
    int j = lane;
    for (; j + 96 < n; j += 128) {
        const unsigned long long k0 = sd.scr.key[j], k1 = sd.scr.key[j + 32];
        const unsigned long long k2 = sd.scr.key[j + 64], k3 = sd.scr.key[j + 96];
        if (k0 < kc && k0 > best) best = k0;
        if (k1 < kc && k1 > best) best = k1;
        if (k2 < kc && k2 > best) best = k2;
        if (k3 < kc && k3 > best) best = k3;
    }
    for (; j < n; j += 32) {
        const unsigned long long k = sd.scr.key[j];
        if (k < kc && k > best) best = k;
    }
    best = warp_max_u64(best);
    return best ? (int)(best & 0xffffffffu) : -1;
}

/* Face walk: point w needs the stencil state left by the last point before it in sort order that
 * made a writer call.  Walk back through the sort order: a done writer gives its record; a done
 * non-writer passes the search to its predecessor; a point not yet done takes w as its waiter and
 * queues it again when it finishes (a point has at most one waiter: waiters lie between it and the
 * next pending point).  Before the face's first point the state is the one the face started with.
 * Keys fall along the walk, so waits cannot form a cycle.  One warp; true with the state when found. */
FD_COLD bool resume_waiter(const fd_station_dev &sd, Shared &sh, int w, float *st0, float *st4)
{
    const int lane = threadIdx.x & 31;
    int c = w;
    for (int guard = 0; guard <= 2 * sh.n + 2; guard++) {
        const int p = predecessor(sd, sh.n, c, lane);
        int verdict = 0;   /* 0 continue from p, 1 found (t0,t4), 2 waiting, 3 retry p */
        float t0 = sh.carry_t0, t4 = sh.carry_t4;
        if (lane == 0) {
            if (p < 0) {
                verdict = 1;
            } else {
                if (vload(sd.scr.pst[p]) != -2) {
                    const int old = atomicCAS(&sd.scr.pst[p], -1, w);
                    if (old == -1) verdict = 2;
                    else if (old == -2) verdict = 3;
                    else { atomicCAS(&sh.w.status, 0, 11); verdict = 2; }   /* a second waiter */
                }
                if (verdict == 0 || verdict == 3) {
                    wfence(sh);
                    const float r0 = vload(sd.scr.rec[p].x), r4 = vload(sd.scr.rec[p].y);
                    if (!isnan(r0)) { verdict = 1; t0 = r0; t4 = r4; }
                    else verdict = 0;
                }
            }
        }
        verdict = __shfl_sync(0xffffffffu, verdict, 0);
        if (verdict == 2) return false;
        if (verdict == 1) {
            *st0 = __shfl_sync(0xffffffffu, t0, 0);
            *st4 = __shfl_sync(0xffffffffu, t4, 0);
            return true;
        }
        c = p;
    }
    if (lane == 0) atomicCAS(&sh.w.status, 0, 12);
    return false;
}

/* nodes of instances not complete that keys_above looks through; with more it waits for the event.  500 windows of 41
 * to 301 a side: 6.42 s without the bound, 6.32 with it at 65536, 6.27 at 131072, 7.97 with no limit; 150 windows of
 * 73 to 91: 319 to 335 ms without, 242 at 65536, 242 and 290 (two models) at 131072, 257 at 16384. */
#ifndef FD_PHI_NODES
#define FD_PHI_NODES 65536
#endif

/* every trial's value is at least the time of one of the node's six neighbours, as the trial reads it: the corner,
 * new-edge and 2-D stencils and the new face reject a value below their times (of the 2-D slots, 1 to 3 are the
 * trial's own), and a 1-D trial adds to one (slownesses are not negative, as the floors of the 1-D trials assume) */
constexpr bool trials_above_a_neighbour()
{
    for (int f = 0; f < FDN_NFACE; f++)
        for (int k = 0; k < FDN_NTRIAL; k++) {
            const fdn_trial tr = fd_face_trials[f][k];
            const int from = tr.kind == FDN_2D ? 1 : 0;
            const int to = tr.kind == FDN_3D ? 7 : tr.kind == FDN_2D ? 4 : tr.kind == FDN_1D ? 1 : 5;
            bool some = false;
            for (int i = from; i < to; i++) {
                const fdn_node n = tr.t[i];
                some = some || n.du * n.du + n.dv * n.dv + n.w * n.w == 1;
            }
            if (!some) return false;
        }
    return true;
}
static_assert(trials_above_a_neighbour(), "keys_above");

/* what a look through the open nodes (not done) of earlier instances found: see keys_above and exit_floor */
struct OpenScan {
    float phi;    /* the least time at the open nodes and their six neighbours (of instance wide: 26) */
    int below;    /* the node with the largest such time that is not above thr, -1 if none is */
    int of_wide;  /* a node of instance wide that is open, -1 if none is */
};

/* the open nodes of the instances before I; false if they are too many to look through */
FD_COLD bool scan_open(const fd_station_dev &sd, Shared &sh, WarpSmem &ws, int I, int wide, float thr, OpenScan &out)
{
    const int lane = threadIdx.x & 31;
    const GraphSmem gs = gsmem(sh);
    unsigned *bits = reinterpret_cast<unsigned *>(&ws.res[0][0]);
    constexpr int kBits = 8 * sizeof ws.res;   /* a flag per node of an instance; larger faces wait for the event */
    if (vload_warp(sh.w.nphi) >= FD_GPHI_CAP - FD_WARPS) return false;   /* these waits leave the tables' room for the others */
    float phi = 1.e10f, worst = -2.f;
    int zw = -1, zj = -1, scanned = 0;
    for (int J0 = 0; J0 < I; J0 += 32) {
        /* the instances that have nodes to come */
        const int Jl = J0 + lane;
        unsigned open = __ballot_sync(0xffffffffu, Jl < I && vload(gs.ndone[Jl < I ? Jl : 0]) < rect_n(gs.rect[Jl < I ? Jl : 0]));
        for (; open; open &= open - 1) {
            const int J = J0 + __ffs(open) - 1;
            const GRect r = gs.rect[J];
            const int n = rect_n(r), nuf = r.nuf();
            scanned += n;
            if (n > kBits || scanned > FD_PHI_NODES) return false;
            const fdn_frame fr = frame_of(r.face());
            const int su = (int)t_stride(sd, fr.axis_u), sv = (int)t_stride(sd, fr.axis_v);
            const int du = 32 % nuf, step = du * su + 32 / nuf * sv, wrap = sv - nuf * su;
            unsigned any = 0;
            int u = lane % nuf, q = inst_node(sd, r, 0) + u * su + lane / nuf * sv;
            for (int j0 = 0; j0 < n; j0 += 128) {
                unsigned c[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    c[k] = j0 + 32 * k + lane < n ? vload(sd.scr.gcnt[q]) : FD_DONEB;
                    u += du;
                    q += step;
                    if (u >= nuf) {
                        u -= nuf;
                        q += wrap;
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned m = __ballot_sync(0xffffffffu, !(c[k] & FD_DONEB));
                    if (lane == 0 && j0 + 32 * k < n) bits[(j0 >> 5) + k] = m;
                    any |= m;
                }
            }
            __syncwarp();
            wfence(sh);
            for (int j0 = 0; any && j0 < n; j0 += 32) {
                if (!((bits[j0 >> 5] >> lane) & 1u)) continue;
                const int xyz = inst_xyz(r, j0 + lane);
                const int x = xyz & 1023, y = (xyz >> 10) & 1023, z = xyz >> 20;
                const int nx = sd.g.nx, nxy = nx * sd.g.ny, p = z * nxy + y * nx + x;
                const int xl = x > 0 ? -1 : 0, xh = x < nx - 1 ? 1 : 0, yl = y > 0 ? -nx : 0, yh = y < sd.g.ny - 1 ? nx : 0;
                const int zl = z > 0 ? -nxy : 0, zh = z < sd.g.nz - 1 ? nxy : 0;
                const int o[7] = {0, xl, xh, yl, yh, zl, zh};
                float lb = 1.e10f;
                float t[7];
#pragma unroll
                for (int k = 0; k < 7; k++) t[k] = sd.T[p + o[k]];
#pragma unroll
                for (int k = 0; k < 7; k++) lb = t[k] >= 0.f ? fminf(lb, t[k]) : -1.f;
                if (J == wide) {
                    for (int k = 0; k < 27; k++) {
                        const float tk = sd.T[p + (k % 3 == 0 ? xl : k % 3 == 2 ? xh : 0) + (k / 3 % 3 == 0 ? yl : k / 3 % 3 == 2 ? yh : 0)
                                              + (k / 9 == 0 ? zl : k / 9 == 2 ? zh : 0)];
                        lb = tk >= 0.f ? fminf(lb, tk) : -1.f;
                    }
                    zj = p;
                }
                phi = fminf(phi, lb);
                if (lb <= thr && lb > worst) {
                    worst = lb;
                    zw = p;
                }
            }
            __syncwarp();
        }
    }
    for (int o = 16; o; o >>= 1) phi = fminf(phi, __shfl_xor_sync(0xffffffffu, phi, o));
    const unsigned m = __reduce_max_sync(0xffffffffu, zw < 0 ? 0u : okey32(worst));
    const unsigned at = __ballot_sync(0xffffffffu, zw >= 0 && okey32(worst) == m);
    out.phi = phi;
    out.below = at ? __shfl_sync(0xffffffffu, zw, __ffs(at) - 1) : -1;
    out.of_wide = (int)__reduce_max_sync(0xffffffffu, zj);
    return true;
}

/* point w waits for open node p, found by scan_open; false if p is done already */
__device__ bool wait_open(const fd_station_dev &sd, Shared &sh, int w, int p)
{
    bool waits = false;
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sh.w.nphi, 1);
        waits = wait_point(sd, sh, w, p);
    }
    return __shfl_sync(0xffffffffu, waits, 0);
}

/* Whether every key of instance I that is not known yet is certainly above kw, so that the points before point w
 * (key kw) are all known already; if not, w is registered on a node that stands against it, or on the event
 * that all keys are known.  One warp.
 *
 * A missing key is the time of a node of an earlier instance that is not done.  Let S be all such nodes and phi
 * the least time now at any of them or their six neighbours: no node of S ends below phi.  For take the first one,
 * in the reference's order, that did: its old time is not below phi, and each trial's value is not below the time
 * it reads at one of the six (trials_above_a_neighbour), which was done before (as read here), is of S and before it
 * (not below phi, since it is the first), or is of an instance not before its own (not changed before it is
 * evaluated).  The flags of an instance are all read before the times about its nodes, and instances go in
 * order: a neighbour whose flag says done then has its final time.  A time that is no number or negative stands
 * against everything.
 *
 * Why: without it such a point waits for the whole inner layer, and where border points inherit state (a fast layer
 * at the grid's edge) the planes of a forward sweep run one after another, which made a few windows five times
 * as long as the others.  Their batches and lists end with them: 150 windows of 73 to 91 319 -> 242 ms, 24 host
 * stations of 49x45x33 96 -> 60, 48 served requests 91 -> 76; with all 26 neighbours instead of the six 251, 65 and 83. */
FD_COLD bool keys_above(const fd_station_dev &sd, Shared &sh, WarpSmem &ws, int I, int w, float kw)
{
    if (vload_warp(sd.scr.ginst[I].phi) > kw) return true;
    OpenScan o;
    for (int turn = 0; turn < 8 && scan_open(sd, sh, ws, I, -1, kw, o); turn++) {   /* a turn more if the node is done by now */
        if (o.phi > kw) {
            if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(&sd.scr.ginst[I].phi), __float_as_int(o.phi));
            return true;
        }
        if (o.below >= 0 && wait_open(sd, sh, w, o.below)) return false;
    }
    if ((threadIdx.x & 31) == 0) wait_event(sd, sh, w, I, 1);
    return false;
}

/* Point w of instance I inherits the state of the last writer of instance J, which is not complete.  A floor of
 * that state's larger time: the last writer is the last one that is done, whose record is there, or a node of J that
 * is open now, and the times of the nodes about that one, when it is evaluated, are not below the least now at any open
 * node before I, its six neighbours and, for J, its 26 (see keys_above).  A floor above the value that won
 * without one (thr) is worth another look at the point: 1, with the floor.  Else it waits for an open node that stands
 * against that (0), or is to wait for J (2).  Such points come first in their instance, where the state is that of
 * the times J ends with, far above their own; waiting for J made the planes of the slowest windows run one after another:
 * 400 windows of 25 to 61 166 and 143 ms (two models) -> 141 and 119, 48 served requests 76 and 50 -> 60 and 38. */
FD_COLD int exit_floor(const fd_station_dev &sd, Shared &sh, WarpSmem &ws, int I, int J, int w, float thr, float *floor)
{
    const GRect rj = gsmem(sh).rect[J];
    OpenScan o;
    for (int turn = 0; turn < 8 && scan_open(sd, sh, ws, I, J, thr, o); turn++) {
        wfence(sh);
        /* after the flags: a point whose flag says done has put its key there (and its record: graph_record) */
        const unsigned long long ek = vload_warp(sd.scr.ginst[J].exitkey);
        if (!ek || !FD_OK((long long)(ek & 0xffffffffu), rect_n(rj), 31)) return 2;
        const int p = inst_node(sd, rj, (int)(ek & 0xffffffffu));
        const float f = fminf(o.phi, fmaxf(vload_warp(sd.scr.grec[p].x), vload_warp(sd.scr.grec[p].y)));
        if (f > thr) {
            if ((threadIdx.x & 31) == 0) atomicAdd(&sh.w.nphi, 1);   /* it may come back to the queue */
            *floor = f;
            return 1;
        }
        const int z = o.below >= 0 ? o.below : o.of_wide;
        if (z < 0) return 2;
        if (wait_open(sd, sh, w, z)) return 0;
    }
    return 2;
}

/* Sweep graph: the same search for point w (packed coordinates), by the reference's order of face
 * instances and, within one, of keys.  Registers w on an instance event or a point when the
 * answer is not yet known.  One warp; true with the state and w's face when found. */
FD_COLD bool resume_graph(const fd_station_dev &sd, Shared &sh, WarpSmem &ws, int w, float *st0, float *st4, bool *floor_only,
                          int *face)
{
    const int lane = threadIdx.x & 31;
    const GraphSmem gs = gsmem(sh);
    const int wx = w & 1023, wy = (w >> 10) & 1023, wz = w >> 20;
    const int ow = owner_of(gs, wx, wy, wz);
    if (ow < 0) {
        if (lane == 0) atomicCAS(&sh.w.status, 0, 14);
        return false;
    }
    const int I = own_inst(ow);
    const GRect r = gs.rect[I];
    const int n = rect_n(r), nuf = r.nuf();
    const fdn_frame fr = frame_of(r.face());
    const int su = (int)t_stride(sd, fr.axis_u), sv = (int)t_stride(sd, fr.axis_v);
    const int base = inst_node(sd, r, 0), in = fr.inner * (int)t_stride(sd, fr.axis_n);
    const int wu = coord(fr.axis_u, wx, wy, wz) - r.ulo, wv = coord(fr.axis_v, wx, wy, wz) - r.vlo;
    const float tw = vload_warp(sd.T[base + wu * su + wv * sv + in]);   /* final: w has been evaluated once */
    if (vload_warp(gs.nkeyed[I]) < n && !keys_above(sd, sh, ws, I, w, tw)) return false;
    wfence(sh);   /* the keys are read after the count, or the bound, that says they are there */
    const unsigned long long kc = node_key(tw, wv * nuf + wu);
    const int dv = 32 / nuf, du = 32 - dv * nuf;   /* 32 points on in fill order */
    for (int guard = 0; guard <= 2 * n + 2; guard++) {
        /* among the instance's earlier points: the last writer that is done, and the last point that is
         * not (it may yet be a writer); four points a lane at a time, so that their loads overlap */
        unsigned long long done = 0ull, pend = 0ull;
        int v = lane / nuf, u = lane - v * nuf;
        for (int j0 = lane; j0 < n; j0 += 128) {
            int q[4];
            unsigned long long key[4];
            unsigned cnt[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                q[k] = base + u * su + v * sv;
                const int j = j0 + 32 * k;
                key[k] = j < n ? node_key(sd.T[q[k] + in], j) : ~0ull;   /* final: every key is */
                u += du;
                v += dv;
                if (u >= nuf) { u -= nuf; v++; }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) cnt[k] = key[k] < kc ? vload(sd.scr.gcnt[q[k]]) : 0u;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (key[k] >= kc) continue;
                if (!(cnt[k] & FD_DONEB)) pend = key[k] > pend ? key[k] : pend;
                else if (cnt[k] & FD_WRITERB) done = key[k] > done ? key[k] : done;
            }
        }
        done = warp_max_u64(done);
        pend = warp_max_u64(pend);
        int verdict = 0;   /* 0 look again, 1 found, 2 waiting, 3 an earlier instance is not complete */
        int before = -1;   /* that instance */
        float t0 = sh.carry_t0, t4 = sh.carry_t4;
        if (lane == 0) {
            if (pend > done) {
                if (wait_point(sd, sh, w, inst_node(sd, r, (int)(pend & 0xffffffffu)))) verdict = 2;
            } else if (done) {
                const long long p = inst_node(sd, r, (int)(done & 0xffffffffu));
                if (!FD_OK((long long)(done & 0xffffffffu), n, 21)) {
                    verdict = 2;
                } else {
                    wfence(sh);
                    verdict = 1;
                    t0 = vload(sd.scr.grec[p].x);
                    t4 = vload(sd.scr.grec[p].y);
                }
            } else {
                /* no writer before it in the instance: the last writer of an earlier instance */
                verdict = 1;
                for (int J = I - 1; J >= 0; J--) {
                    const GRect &rj = gs.rect[J];
                    if (vload(gs.ndone[J]) < rect_n(rj)) { before = J; verdict = 3; break; }
                    wfence(sh);
                    const unsigned long long ek = vload(sd.scr.ginst[J].exitkey);
                    if (ek) {
                        const long long p = inst_node(sd, rj, (int)(ek & 0xffffffffu));
                        if (!FD_OK((long long)(ek & 0xffffffffu), rect_n(rj), 22)) break;
                        t0 = vload(sd.scr.grec[p].x);
                        t4 = vload(sd.scr.grec[p].y);
                        break;
                    }
                }
            }
        }
        verdict = __shfl_sync(0xffffffffu, verdict, 0);
        if (verdict == 3) {
            before = __shfl_sync(0xffffffffu, before, 0);
            float f = 0.f;
            const int can = exit_floor(sd, sh, ws, I, before, w, vload_warp(sd.scr.grec[node_of(sd, w)].x), &f);
            if (can == 1) {
                *st0 = *st4 = f;
                *floor_only = true;
                *face = r.face();
                return true;
            }
            if (can == 2 && lane == 0) wait_event(sd, sh, w, before, 2);
            return false;
        }
        if (verdict == 2) return false;
        if (verdict == 1) {
            *st0 = __shfl_sync(0xffffffffu, t0, 0);
            *st4 = __shfl_sync(0xffffffffu, t4, 0);
            *face = r.face();
            return true;
        }
    }
    if (lane == 0) atomicCAS(&sh.w.status, 0, 12);
    return false;
}

/* ---------------------------------------------------------------------------------------------- */
/* the worker loop                                                                                 */

/* nothing queued, every worker idle, and all queues unchanged across the idle count (lane 0) */
__device__ __forceinline__ bool quiescent(Shared &sh)
{
    int t0[6], r0 = vload(sh.w.rqtail);
    for (int k = 0; k < sh.w.nq; k++) {
        t0[k] = vload(sh.w.qtail[k]);
        if (vload(sh.w.qhead[k]) != t0[k]) return false;
    }
    if (vload(sh.w.rqhead) != r0) return false;
    wfence(sh);
    if (vload(sh.w.idle) != FD_WARPS) return false;
    wfence(sh);
    for (int k = 0; k < sh.w.nq; k++)
        if (vload(sh.w.qtail[k]) != t0[k] || vload(sh.w.qhead[k]) != t0[k]) return false;
    return vload(sh.w.rqtail) == r0 && vload(sh.w.rqhead) == r0;
}

/* read a claimed queue entry: spins briefly for an entry whose writer is between its two
 * instructions; -1 and a status on failure */
__device__ __forceinline__ int read_entry(const int *queue, int pos, Shared &sh)
{
    const volatile int *q = queue + pos;
    int e = *q;
    for (int spin = 0; e < 0 && spin < FD_QSPIN; spin++) {
        __nanosleep(32);
        e = *q;
    }
    if (e < 0) atomicCAS(&sh.w.status, 0, 9);   /* a claimed entry never written */
    return e;
}

/* the worker loop of one walk over `total` nodes; all warps call it between two CTA barriers */
__device__ void run_walk(const fd_station_dev &sd, Shared &sh, const CtaSmem &cs, WarpSmem &ws, int total,
                         unsigned char *dag, Counters cn)
{
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int *queue = sh.graph ? sd.scr.gqueue : sd.scr.queue;
    int *rq = sh.graph ? sd.scr.grq : sd.scr.rq;
    bool idle = false;
    long long since = clock64();
    const long long started = since;
    const long long wait_lim = sd.wait_cycles > 0 ? sd.wait_cycles : FD_WAIT_CYCLES;
    const long long walk_lim = sd.walk_cycles > 0 ? sd.walk_cycles : FD_WALK_CYCLES;
    long long chunks = 0;
    unsigned idle_polls = 0;
    for (;;) {
        /* One look at all counters, a queue per lane (0-5 ready nodes by face, 6 resuming points): what every
         * chunk of a latency-bound sweep waits for, so it is kept to a few dozen instructions (a
         * loop over the queues in lane 0 took about 400). */
        int hd = 0, avail = 0;
        bool stop = false;
        if (lane < 6) {
            hd = vload(sh.w.qhead[lane]);
            const int qt = vload(sh.w.qtail[lane]);
            avail = min(qt, sh.w.qcap[lane]) - hd;
        } else if (lane == 6) {
            hd = vload(sh.w.rqhead);
            const int qt = vload(sh.w.rqtail);
            avail = min(qt, sh.w.rqcap) - hd;
        } else if (lane == 7) {
            stop = vload(sh.w.status) != 0 || vload(sh.w.ndone) >= total;
        }
        if (__any_sync(0xffffffffu, stop)) break;
        /* resuming points first, else the fullest queue, ties in a warp-dependent order */
        const int pref = avail <= 0 ? 0 : lane == 6 ? 0x7fffffff : lane < 6 ? avail << 3 | ((lane + warp) & 7) : 0;
        const int best = __reduce_max_sync(0xffffffffu, pref);
        int act = 0, h = 0, m = 0, qf = 0;   /* act: 0 nothing, 1 chunk, 2 resume a waiter */
        if (best) {
            qf = __ffs(__ballot_sync(0xffffffffu, pref == best)) - 1;
            if (idle && lane == 0) atomicSub(&sh.w.idle, 1);
            idle = false;
            if (lane == qf) {
                m = lane == 6 ? 1 : min(avail, 32);
                int *head = lane == 6 ? &sh.w.rqhead : &sh.w.qhead[lane];
                if (atomicCAS(head, hd, hd + m) == hd) act = lane == 6 ? 2 : 1;
                h = lane == 6 ? hd : sh.w.qbase[lane] + hd;
            }
            act = __shfl_sync(0xffffffffu, act, qf);
            h = __shfl_sync(0xffffffffu, h, qf);
            m = __shfl_sync(0xffffffffu, m, qf);
        } else {
            if (!idle) {
                wfence(sh);
                if (lane == 0) atomicAdd(&sh.w.idle, 1);
                idle = true;
                idle_polls = 0;
            }
            /* all idle with nothing queued and nodes left: nothing can release them.  The
             * check (two fences and a scan of every queue) runs on every 64th idle poll
             * only: idle warps are most of the CTA in a forward sweep, and their polls
             * share the SM's shared-memory pipe with the working warps */
            if ((++idle_polls & 63u) == 0u && lane == 0 && quiescent(sh) && vload(sh.w.ndone) < total)
                atomicCAS(&sh.w.status, 0, 3);
        }
        if (lane == 0) {
            const long long now = clock64();
            if (act) since = now;
            else if (now - since > wait_lim) atomicCAS(&sh.w.status, 0, 8);   /* no work for this worker for too long */
            if (now - started > walk_lim) atomicCAS(&sh.w.status, 0, 17);     /* the walk as a whole ran far too long */
        }
        if (!act) {
            if (!best) __nanosleep(64);
            continue;
        }
        int e = -1, face = sh.face;
        float in0 = 0.f, in4 = 0.f;
        bool floor_only = false;
        if (lane < m) {
            e = read_entry((act == 1 ? queue : rq) + h, lane, sh);
            /* an entry outside the walk's nodes ends the walk with a status instead of an access */
            const bool ok = sh.graph ? (e & 1023) < sd.g.nx && ((e >> 10) & 1023) < sd.g.ny && (e >> 20) < sd.g.nz : e < sh.n;
            if (e >= 0 && !ok) {
                (void)FD_OK(e, 0, 23);
                atomicCAS(&sh.w.status, 0, 18);
                e = -1;
            }
        }
        wfence(sh);
        if (act == 1) {
            if (sh.graph) face = qf;
            chunks++;
        } else {
            h = __shfl_sync(0xffffffffu, e, 0);
            if (h < 0 || !(sh.graph ? resume_graph(sd, sh, ws, h, &in0, &in4, &floor_only, &face) : resume_waiter(sd, sh, h, &in0, &in4))) continue;
        }
        warp_chunk(sd, sh, cs, ws, face, e, act == 2 ? (floor_only ? kFloor : kState) : kNoState, in0, in4, dag, cn);
    }
    if (lane == 0 && chunks) atomicAdd(reinterpret_cast<unsigned long long *>(&sh.w.rounds), (unsigned long long)chunks);
}

/* reset the walk counters (thread 0) */
__device__ void walk_reset(Shared &sh, int nq, int rqcap)
{
    sh.w.nq = nq;
    for (int k = 0; k < 6; k++) { sh.w.qhead[k] = 0; sh.w.qtail[k] = 0; sh.w.qcap[k] = 0; sh.w.qbase[k] = 0; }
    sh.w.rqhead = sh.w.rqtail = sh.w.idle = sh.w.ndone = sh.w.npark = sh.w.nphi = 0;
    sh.w.rqcap = rqcap;
    sh.w.exitkey = 0ull;
}

/* Walk the current face (parameters in sh) in dependency order. */
__device__ void face_walk(const fd_station_dev &sd, Shared &sh, CtaSmem &cs, WarpSmem &ws, unsigned char *dag,
                          Counters cn)
{
    const int n = sh.n, nuf = sh.nuf, nvf = n / nuf;
    const int tid = threadIdx.x;
    const float *T = sd.T;
    const fdn_frame fr = frame_of(sh.face);
    unsigned char *emask = dag + sh.n_pad;
    int *queue = sd.scr.queue;
    FD_TIC(t0);
    /* keys: time of the inner-layer neighbour, then fill index */
    for (int i = tid; i < n; i += blockDim.x) {
        int x, y, z;
        place(fr, sh.ulo + i % nuf, sh.vlo + i / nuf, sh.layer + fr.inner, x, y, z);
        const float tin = T[((long long)z * sd.g.ny + y) * sd.g.nx + x];
        sd.scr.key[i] = ((unsigned long long)okey32(tin) << 32) | (unsigned)i;
        sd.scr.pst[i] = -1;
        queue[i] = -1;
        sd.scr.rq[2 * i] = -1;
        sd.scr.rq[2 * i + 1] = -1;
    }
    if (tid == 0) {
        walk_reset(sh, 1, 2 * n);
        sh.w.qcap[0] = n;
        sh.graph = 0;
    }
    __syncthreads();
    /* earlier-neighbour masks and in-degrees */
    for (int i = tid; i < n; i += blockDim.x) {
        const unsigned long long ki = sd.scr.key[i];
        const int iu = i % nuf, iv = i / nuf;
        unsigned em = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            int du, dv;
            nb_off(k, du, dv);
            const int ju = iu + du, jv = iv + dv;
            if (ju < 0 || ju >= nuf || jv < 0 || jv >= nvf) continue;
            if (sd.scr.key[jv * nuf + ju] < ki) em |= 1u << k;
        }
        emask[i] = (unsigned char)em;
        dag[i] = (unsigned char)__popc(em);
        if (em == 0) enqueue_to(queue, sh.w.qtail[0], sh.w.qcap[0], sh, i);
    }
    __syncthreads();
    FD_TOC(0, t0);
    FD_TIC(tw);
    run_walk(sd, sh, cs, ws, n, dag, cn);
    __syncthreads();
    FD_TOC(4, tw);
    if (tid == 0) {
        if (sh.w.exitkey) {
            const float2 r = sd.scr.rec[(int)(sh.w.exitkey & 0xffffffffu)];
            sh.carry_t0 = r.x;
            sh.carry_t4 = r.y;
        }
        sh.faces++;
        sh.node_updates += n;
    }
}

/* face parameters of face `face` for the current walls (thread 0) */
__device__ void setup_face(Shared &sh, int face)
{
    /* walls: 0 z1, 1 z2, 2 x2, 3 x1, 4 y1, 5 y2 */
    const int x1 = sh.wall[3], x2 = sh.wall[2], y1 = sh.wall[4], y2 = sh.wall[5];
    const int z1 = sh.wall[0], z2 = sh.wall[1];
    sh.face = face;
    sh.layer = sh.wall[face];
    if (face < 2) {
        sh.ulo = x1 + 1; sh.uhi = x2 - 1; sh.vlo = y1 + 1; sh.vhi = y2 - 1;
    } else if (face < 4) {
        sh.ulo = y1 + 1; sh.uhi = y2 - 1; sh.vlo = z1 + 1; sh.vhi = z2 - 1;
    } else {
        sh.ulo = x1 + 1; sh.uhi = x2 - 1; sh.vlo = z1 + 1; sh.vhi = z2 - 1;
    }
    sh.nuf = sh.uhi - sh.ulo + 1;
    const int nvf = sh.vhi - sh.vlo + 1;
    sh.n = (sh.nuf > 0 && nvf > 0) ? sh.nuf * nvf : 0;
    sh.n_pad = (sh.n + 15) & ~15;
}

/* One sweep (the radius loop of src/sphfd.c:1018-5566) as one dependency graph.  Leaves walls,
 * flags, radius and the stencil-state carry as the radius loop would. */
__device__ void graph_sweep(const fd_station_dev &sd, Shared &sh, CtaSmem &cs, WarpSmem &ws, Counters cn)
{
    const int tid = threadIdx.x;
    const int nx = sd.g.nx, ny = sd.g.ny, nz = sd.g.nz;
    const GraphSmem gs = gsmem(sh);
    FD_TIC(t0);
    /* walls: 0 z1, 1 z2, 2 x2, 3 x1, 4 y1, 5 y2 */
    for (int k = tid; k < sh.lstride; k += blockDim.x) {
        const int c = k - 1;
        gs.lay[0][k] = c >= 0 && c < nx && c > sh.wall[3] && c < sh.wall[2] ? FD_IN_BOX : FD_NEVER;
        gs.lay[1][k] = c >= 0 && c < ny && c > sh.wall[4] && c < sh.wall[5] ? FD_IN_BOX : FD_NEVER;
        gs.lay[2][k] = c >= 0 && c < nz && c > sh.wall[0] && c < sh.wall[1] ? FD_IN_BOX : FD_NEVER;
    }
    __syncthreads();
    /* the sweep's face instances, as the radius loop visits them */
    if (tid == 0) {
        const int cap = sd.scr.ginst_cap < sh.imax ? sd.scr.ginst_cap : sh.imax;
        int ninst = 0;
        long long M = 0, per_face[6] = {0, 0, 0, 0, 0, 0};
        unsigned faces = 0;
        bool over = false;
        while (sh.rad0 && (sh.dflag[0] || sh.dflag[1] || sh.dflag[2] || sh.dflag[3] || sh.dflag[4] || sh.dflag[5])) {
            for (int face = 0; face < 6; face++) {
                for (int ig = 1; ig <= sd.grow[face]; ig++) {
                    if (!sh.dflag[face]) continue;
                    setup_face(sh, face);
                    if (sh.n > 0) {
                        if (ninst >= cap) { over = true; break; }
                        fd_ginst &gi = sd.scr.ginst[ninst];
                        gi.phi = 0.f;
                        gi.ev[0] = gi.ev[1] = FD_EV_NONE; gi.exitkey = 0ull;
                        GRect &gr = gs.rect[ninst];
                        gr.fl = (short)(sh.layer << 3 | face);
                        gr.ulo = (short)sh.ulo; gr.uhi = (short)sh.uhi; gr.vlo = (short)sh.vlo; gr.vhi = (short)sh.vhi;
                        gs.nkeyed[ninst] = 0;
                        gs.ndone[ninst] = 0;
                        gs.lay[frame_of(face).axis_n][sh.layer + 1] = (short)((ninst << 3) | face);
                        ninst++;
                        M += sh.n;
                        per_face[face] += sh.n;
                        faces |= 1u << face;
                    } else {
                        /* a wall that moves while its rectangle is empty owns no node: its nodes join
                         * with a later wall, and any word between the instances around it does */
                        gs.lay[frame_of(face).axis_n][sh.layer + 1] = (short)(((ninst - 1) << 3) | 7);
                    }
                    /* move the wall outward (e.g. src/sphfd.c:1762-1764) */
                    const int inner = frame_of(face).inner;
                    const int nmax = face < 2 ? nz : face < 4 ? nx : ny;
                    const bool limit = inner > 0 ? (sh.wall[face] == 0) : (sh.wall[face] == nmax - 1);
                    if (limit) sh.dflag[face] = 0;
                    sh.wall[face] -= inner;
                }
            }
            sh.radius++;
            if (sh.radius == sd.maxrad) sh.rad0 = 0;
            if (over) break;
        }
        sh.ninst = ninst;
        sh.gfaces = faces;
        sh.single = __popc(faces) == 1;
        sh.nodefer = 0;
        sh.graph = 1;
        sh.gM = M;
        if (over) sh.w.status = 13;
        walk_reset(sh, 6, FD_GRQ_CAP);
        sh.w.nwait = 0;
        long long b = 0;
        for (int f = 0; f < 6; f++) { sh.w.qbase[f] = (int)b; sh.w.qcap[f] = (int)per_face[f]; b += per_face[f]; }
    }
    csync(sh);
    const int ninst = sh.ninst;
    const long long M = sh.gM;
    if (sh.single) {
        /* One face, every time below 1e9: every corner guard inside the grid passes, so each point
         * calls a corner stencil before its 2-D trials and none needs an earlier point's state;
         * the exception is the EAST corner whose guard tests the node above for being non-zero
         * (src/sphfd.c:2544), which fails only next to a zero time. */
        const int f = __ffs(sh.gfaces) - 1;
        const long long nxyz = (long long)nx * ny * nz;
        int bad = 0;
        for (long long q = tid; q < nxyz; q += blockDim.x) {
            const float t = __ldcg(&sd.T[q]);
            if (!(t < 1.e9f)) bad = 1;
            else if (f == 2 && t == 0.0f && (q / nx) % ny == 0 && q / ((long long)nx * ny) == 1) bad = 1;
        }
        bad = __syncthreads_or(bad);
        if (tid == 0) sh.nodefer = !bad;
        __syncthreads();
    }
    if (M > 0 && sh.stat == 0) {
        for (long long k = tid; k < M; k += blockDim.x) sd.scr.gqueue[k] = -1;
        /* dependency counters */
        for (int I = 0; I < ninst; I++) {
            const GRect r = gs.rect[I];
            const fdn_frame fr = frame_of(r.face());
            const int n = rect_n(r), nuf = r.nuf(), nvf = r.vhi - r.vlo + 1;
            const unsigned myctx = sh.ctxm[r.face()], myinn = sh.innm[r.face()];
            const bool prev = sh.single && I > 0 && gs.rect[I - 1].layer() == r.layer() + fr.inner;
            for (int j = tid; j < n; j += blockDim.x) {
                const int xyz = inst_xyz(r, j), p = node_of(sd, xyz);
                if (!FD_OK(p, (long long)nx * ny * nz, 25)) continue;
                unsigned cin = 0, c2 = 0, cx = 0;
                if (sh.single) {
                    /* one face: the same-instance neighbours and the previous plane's inner block */
                    const int iv = j / nuf, iu = j - iv * nuf;
                    c2 = (unsigned)__popc(inrect_mask(iu, iv, nuf, nvf));
                    if (prev) {
                        const GRect &rp = gs.rect[I - 1];
                        const int u0 = r.ulo + iu, v0 = r.vlo + iv;
                        for (int dv = -1; dv <= 1; dv++)
                            for (int du = -1; du <= 1; du++)
                                if (u0 + du >= rp.ulo && u0 + du <= rp.uhi && v0 + dv >= rp.vlo && v0 + dv <= rp.vhi) cin++;
                    }
                } else {
                    const int x = xyz & 1023, y = (xyz >> 10) & 1023, z = xyz >> 20;
                    int lx[3], ly[3], lz[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        lx[k] = gs.lay[0][x + k];
                        ly[k] = gs.lay[1][y + k];
                        lz[k] = gs.lay[2][z + k];
                    }
#pragma unroll
                    for (int k = 0; k < 27; k++) {
                        if (k == 13) continue;
                        const int w = owner_word(lx[k % 3], ly[(k / 3) % 3], lz[k / 9]);
                        if (w < 0 || own_inst(w) > I) continue;
                        if (own_inst(w) == I) { c2++; continue; }
                        if (!((myctx >> k) & 1u) && !((sh.ctxm[own_face(w)] >> (26 - k)) & 1u)) continue;
                        if ((myinn >> k) & 1u) cin++; else cx++;
                    }
                }
                sd.scr.gcnt[p] = cin | (c2 << 8) | (cx << 16);
            }
        }
        csync(sh);
        /* nodes whose inner block is final take their key now */
        for (int I = 0; I < ninst; I++) {
            const GRect r = gs.rect[I];
            const int n = rect_n(r);
            for (int j = tid; j < n; j += blockDim.x) {
                const int xyz = inst_xyz(r, j), p = node_of(sd, xyz);
                if ((sd.scr.gcnt[p] & 0xFFu) == 0u && ready_word(key_event(sd, sh, I, xyz, p))) graph_ready(sd, sh, r.face(), xyz);
            }
        }
        csync(sh);
        FD_TOC(0, t0);
        FD_TIC(tw);
        run_walk(sd, sh, cs, ws, (int)M, nullptr, cn);
        csync(sh);
        FD_TOC(4, tw);
    }
    /* the small tables back to their empty state for the next sweep */
    {
        const int nw = vload(sh.w.nwait) > 0 ? FD_GWAIT_CAP : 0;
        const int nr = min(vload(sh.w.rqtail), FD_GRQ_CAP);
        for (int k = tid; k < nw; k += blockDim.x) sd.scr.gwait[k] = make_int2(-1, -1);
        for (int k = tid; k < nr; k += blockDim.x) sd.scr.grq[k] = -1;
    }
    if (tid == 0) {
        /* the stencil state after the sweep: the record of its last writer */
        for (int I = ninst - 1; I >= 0; I--) {
            const unsigned long long ek = vload(sd.scr.ginst[I].exitkey);
            if (ek && FD_OK((long long)(ek & 0xffffffffu), rect_n(gs.rect[I]), 26)) {
                const float2 r = __ldcg(&sd.scr.grec[inst_node(sd, gs.rect[I], (int)(ek & 0xffffffffu))]);
                sh.carry_t0 = r.x;
                sh.carry_t4 = r.y;
                break;
            }
        }
        sh.faces += ninst;
        sh.node_updates += M;
        sh.gsweeps++;
        sh.graph = 0;
    }
    csync(sh);
}

/* ---------------------------------------------------------------------------------------------- */

/* source box (src/sphfd.c:724-825)                                                                */

__device__ void init_field(const fd_station_dev &sd)
{
    const long long nxyz = (long long)sd.g.nx * sd.g.ny * sd.g.nz;
    const float u = 1.0e10f;
    /* T may start anywhere a float can: scalar head up to a 16-byte boundary, float4 body, scalar tail */
    const long long head = (long long)(((16u - ((unsigned)(uintptr_t)sd.T & 15u)) & 15u) / 4u);
    const long long h = head < nxyz ? head : nxyz;
    for (long long i = threadIdx.x; i < h; i += blockDim.x) sd.T[i] = u;
    float4 *T4 = reinterpret_cast<float4 *>(sd.T + h);
    const long long nv4 = (nxyz - h) / 4;
    for (long long i = threadIdx.x; i < nv4; i += blockDim.x) T4[i] = make_float4(u, u, u, u);
    for (long long i = h + nv4 * 4 + threadIdx.x; i < nxyz; i += blockDim.x) sd.T[i] = u;
    __syncthreads();
    const int nc = sd.ncube, w = 2 * nc + 1;
    const long long nx = sd.g.nx, nxy = (long long)sd.g.nx * sd.g.ny;
    const float s000 = sd.S[(long long)sd.zs * sd.s_sz + (long long)sd.ys * sd.s_sy + sd.xs];
    for (int k = threadIdx.x; k < w * w * w; k += blockDim.x) {
        const int zz = sd.zs - nc + k / (w * w), yy = sd.ys - nc + (k / w) % w, xx = sd.xs - nc + k % w;
        if (zz < 0 || zz >= sd.g.nz || yy < 0 || yy >= sd.g.ny || xx < 0 || xx >= sd.g.nx) continue;
        const int jy = yy - (sd.ys - nc), jx = xx - (sd.xs - nc);
        const double cq = sd.box_trig[2 * jy], sq = sd.box_trig[2 * jy + 1];
        const double cf = sd.box_trig[2 * w + 2 * jx], sf = sd.box_trig[2 * w + 2 * jx + 1];
        const double rz1 = sd.g.zrow[(long long)zz * FD_Z_N + FD_Z_R];
        const double x2p = rz1 * cq;
        const double y2p = rz1 * sq * cf;
        const double z2p = rz1 * sq * sf;
        const double dx = sd.src_xyz[0] - x2p, dy = sd.src_xyz[1] - y2p, dz = sd.src_xyz[2] - z2p;
        const double dist = __dsqrt_rn(dx * dx + dy * dy + dz * dz);
        sd.T[(long long)zz * nxy + (long long)yy * nx + xx] = __double2float_rn((double)s000 * dist);
    }
    __syncthreads();
}

/* ---------------------------------------------------------------------------------------------- */
/* the sweep loop (src/sphfd.c:1008-5678)                                                          */

/* The solve of one station by this CTA.  sd is the station record in this CTA's shared memory; lmax and imax
 * are the extent and the instances that the launch's sweep-graph tables have room for. */
__device__ __forceinline__ void solve_station(const fd_station_dev &sd, int dag_smem_bytes, int lmax, int imax, Shared &sh)
{
    extern __shared__ __align__(16) unsigned char fd_dyn_smem[];
    CtaSmem &cs = *reinterpret_cast<CtaSmem *>(fd_dyn_smem);
    WarpSmem &ws = reinterpret_cast<WarpSmem *>(fd_dyn_smem + kCtaSmemBytes)[threadIdx.x >> 5];
    const int tid = threadIdx.x;
    unsigned long long t_start = 0;
    if (tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    /* the dependency bytes of the station's largest face go to shared memory when they fit */
    unsigned char *dag = 2ll * sd.max_face_pad <= dag_smem_bytes ? fd_dyn_smem + kSmemBase : sd.scr.dag;
    const int gdim = sd.g.nx > sd.g.ny ? (sd.g.nx > sd.g.nz ? sd.g.nx : sd.g.nz) : (sd.g.ny > sd.g.nz ? sd.g.ny : sd.g.nz);
    const bool gok = sd.scr.gcnt && gdim <= lmax && sd.scr.ginst_cap <= imax && graph_smem_bytes(lmax, imax) <= dag_smem_bytes;
    if (tid == 0) sh.stat = 0;
    if (gok) {
        /* the sweep-graph tables start empty */
        for (int k = tid; k < FD_GWAIT_CAP; k += blockDim.x) sd.scr.gwait[k] = make_int2(-1, -1);
        for (int k = tid; k < FD_GRQ_CAP; k += blockDim.x) sd.scr.grq[k] = -1;
    }
    if (sd.init_mode == 0) init_field(sd);
    for (int k = tid; k < FDN_NFACE * FDN_NTRIAL; k += blockDim.x) (&cs.desc[0][0])[k] = c_desc[k];
    if (tid == 0) {
        for (int f = 0; f < 6; f++) { sh.wall[f] = sd.wall[f]; sh.dflag[f] = sd.dflag[f]; }
        sh.radius = sd.radius;
        sh.rad0 = 1;
        sh.reverse = sd.reverse;
        sh.headpref = sd.headpref;
        sh.carry_t0 = sd.carry_t0;
        sh.carry_t4 = sd.carry_t4;
        sh.w.status = 0;
        sh.w.rounds = sh.w.deferred = 0;
        for (int k = 0; k < 5; k++) sh.w.st[k] = 0;
        sh.w.nwait = 0;
        sh.w.npark = 0;
        sh.faces = sh.node_updates = 0;
        sh.sweeps = 0;
        for (int k = 0; k < 8; k++) sh.restart_wall[k] = 0;
        for (int k = 0; k < 6; k++) sh.cyc[k] = 0;
        sh.graph = 0;
        sh.gsweeps = 0;
        for (int f = 0; f < 6; f++) relation_masks(f, sh.ctxm[f], sh.innm[f]);
        sh.lstride = lmax + 2;
        sh.imax = imax;
        sh.gok = gok;
        sh.single = 0;
        sh.nodefer = 0;
        sh.gfaces = 0;
    }
    csync(sh);
    for (int k = tid; k < 6 * 27; k += blockDim.x) sh.rel[k / 27][k % 27] = relation_word(sh, k / 27, k % 27);
    if ((tid & 31) < 6) ws.cnt[tid & 31] = 0ull;
    __syncwarp();
    Counters cn;
    cn.n = ws.cnt;
    const int nx = sd.g.nx, ny = sd.g.ny, nz = sd.g.nz;
    int guard_sweeps = 0;
    while (sh.reverse > -1 && sh.stat == 0) {
        if (tid == 0) for (int k = 0; k < 8; k++) sh.w.headw[k] = 0;
        csync(sh);
        FD_TIC(tsweep);
        const bool as_graph = sh.gok && (FD_GRAPH_FORWARD || sh.sweeps > 0);
        if (as_graph) graph_sweep(sd, sh, cs, ws, cn);
        while (!as_graph && sh.rad0
               && (sh.dflag[0] || sh.dflag[1] || sh.dflag[2] || sh.dflag[3] || sh.dflag[4] || sh.dflag[5])
               && sh.stat == 0) {
            for (int face = 0; face < 6; face++) {
                for (int ig = 1; ig <= sd.grow[face]; ig++) {
                    if (!sh.dflag[face]) continue;
                    if (tid == 0) setup_face(sh, face);
                    __syncthreads();
                    if (sh.n > 0) face_walk(sd, sh, cs, ws, dag, cn);
                    __syncthreads();
                    if (tid == 0) {
                        /* move the wall outward (e.g. src/sphfd.c:1762-1764) */
                        const int inner = frame_of(face).inner;
                        const int nmax = face < 2 ? nz : face < 4 ? nx : ny;
                        const bool limit = inner > 0 ? (sh.wall[face] == 0) : (sh.wall[face] == nmax - 1);
                        if (limit) sh.dflag[face] = 0;
                        sh.wall[face] -= inner;
                    }
                    __syncthreads();
                }
            }
            if (tid == 0) {
                sh.radius++;
                if (sh.radius == sd.maxrad) sh.rad0 = 0;
            }
            csync(sh);
        }
        if (tid == 0) {
            if (sh.sweeps == 0) FD_TOC(5, tsweep);   /* profiling builds: the first sweep's cycles */
            sh.sweeps++;
            /* restart test (src/sphfd.c:5570-5676) */
            const int *hw = sh.w.headw;
            if (!hw[1] && !hw[2] && !hw[3] && !hw[4] && !hw[5] && !hw[6]) {
                sh.reverse = 0;
            } else {
                int head = 0, srcwall = 0;
                for (int w = 1; w <= 6; w++)
                    if (hw[w] > 0 && hw[w] > head) { head = hw[w]; srcwall = w; }
                if (sh.headpref > 0 && hw[sh.headpref] > 0) srcwall = sh.headpref;
                for (int f = 0; f < 6; f++) sh.dflag[f] = 1;
                sh.rad0 = 1;
                sh.radius = 1;
                /* face order walls: 0 z1, 1 z2, 2 x2, 3 x1, 4 y1, 5 y2 */
                if (srcwall == 1) sh.wall[2] = 1; else { sh.wall[2] = nx; sh.dflag[2] = 0; }
                if (srcwall == 2) sh.wall[3] = nx - 2; else { sh.wall[3] = -1; sh.dflag[3] = 0; }
                if (srcwall == 3) sh.wall[5] = 1; else { sh.wall[5] = ny; sh.dflag[5] = 0; }
                if (srcwall == 4) sh.wall[4] = ny - 2; else { sh.wall[4] = -1; sh.dflag[4] = 0; }
                if (srcwall == 5) sh.wall[1] = 1; else { sh.wall[1] = nz; sh.dflag[1] = 0; }
                if (srcwall == 6) sh.wall[0] = nz - 2; else { sh.wall[0] = -1; sh.dflag[0] = 0; }
                if (sh.reverse > 0) sh.restart_wall[srcwall]++;
            }
            sh.reverse--;
        }
        csync(sh);
        if (++guard_sweeps > 1000000) { if (tid == 0) sh.w.status = 4; break; }
    }
    /* statistics */
    __syncwarp();
    if ((tid & 31) < 5) atomicAdd(&sh.w.st[tid & 31], ws.cnt[tid & 31]);
    csync(sh);
    if (tid == 0 && sd.stats) {
        fd_station_stats *o = sd.stats;
        o->status = sh.w.status;
        o->sweeps = sh.sweeps;
        o->node_updates = sh.node_updates;
        o->faces = sh.faces;
        o->rounds = sh.w.rounds;
        o->deferred = sh.w.deferred;
        for (int k = 0; k < 5; k++) o->stencils[k] = (int64_t)sh.w.st[k];
        for (int k = 0; k < 8; k++) o->restart_wall[k] = sh.restart_wall[k];
        for (int k = 0; k < 6; k++) o->phase_cycles[k] = sh.cyc[k];
        unsigned long long t_end;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
        o->t_start_ns = (int64_t)t_start;
        o->t_end_ns = (int64_t)t_end;
        o->pipelined_sweeps = (int32_t)sh.gsweeps;
        unsigned smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        o->sm = (int32_t)smid;
    }
}

/* a station record copied into shared memory by the whole CTA; cache-volatile loads, because a
 * serving session rewrites a record slot between the requests this SM reads from it */
__device__ __forceinline__ void load_record(fd_station_dev &dst, const fd_station_dev *src)
{
    static_assert(sizeof(fd_station_dev) % 4 == 0, "record size");
    const unsigned *s = reinterpret_cast<const unsigned *>(src);
    unsigned *d = reinterpret_cast<unsigned *>(&dst);
    for (int k = threadIdx.x; k < (int)(sizeof(fd_station_dev) / 4); k += blockDim.x) d[k] = __ldcv(s + k);
}

__device__ __forceinline__ unsigned long long ld_acquire_sys(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_sys(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

/* Thread 0 claims the next published request of a serving session: its entry, or -1 when the host
 * has asked idle CTAs to stop, or -2 after q.idle_ns with nothing to claim (the host normally
 * stops the grid long before; the bound only ends a loop whose host has gone away). */
__device__ int serve_claim(const fd_serve_queue &q, unsigned long long *gen)
{
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    /* Idle CTAs back off between looks, to 2 us on SM 0 and ~60 us on the last SM: a burst of
     * requests is claimed mostly by the low-numbered SMs, the ones a batch launch of as many CTAs
     * fills first (a 64-station batch lands on SMs 0-59 and 148-151).  Packed that way the same
     * stations solved 14 % faster than spread over both dies. */
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    const unsigned cap_ns = 2000u + 400u * smid;
    unsigned sleep_ns = 500;
    for (;;) {
        const unsigned long long h = *(volatile const unsigned long long *)q.head;
        const unsigned long long t = ld_acquire_sys(q.tail);
        if (h < t) {
            if (atomicCAS(q.head, h, h + 1) == h) {
                const int e = *(volatile const int *)(q.order + (h % (unsigned long long)q.ring));
                *gen = *(volatile const unsigned long long *)(q.gen + e);
                return e;
            }
            continue;
        }
        if (*(volatile const int *)q.stop) return -1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if ((long long)(now - t0) > q.idle_ns) return -2;
        __nanosleep(sleep_ns);
        if (sleep_ns < cap_ns) sleep_ns = sleep_ns * 2 < cap_ns ? sleep_ns * 2 : cap_ns;
    }
}

/* Batch mode (q == nullptr): station blockIdx.x of `stations`, one launch per batch.
 * Serving mode: a long-running grid of one CTA per SM; each CTA solves the requests it claims from
 * q one after another, and writes exitf[cta_id0 + blockIdx.x] when it leaves. */
__global__ void __launch_bounds__(FD_BLOCK, 1) fd_solve(const fd_station_dev *stations, int nst, int dag_smem_bytes,
                                                       int lmax, int imax, const fd_serve_queue *q, int cta_id0)
{
    __shared__ Shared sh;
    __shared__ fd_station_dev rec;
    __shared__ int entry;
    __shared__ unsigned long long gen;
    const int station = (int)blockIdx.x;
    if (!q && station >= nst) return;
    for (;;) {
        if (q) {
            if (threadIdx.x == 0) entry = serve_claim(*q, &gen);
            __syncthreads();
            if (entry < 0) break;
        }
        load_record(rec, q ? q->desc + entry : stations + station);
        __syncthreads();
        solve_station(rec, dag_smem_bytes, lmax, imax, sh);
        if (!q) return;
        /* every thread's field writes, then the statistics, then the flag the host waits for */
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence_system();
            st_release_sys(q->done + entry, gen);
        }
    }
    if (threadIdx.x == 0) {
        __threadfence_system();
        *(volatile int *)(q->exitf + cta_id0 + blockIdx.x) = 1;
    }
}

}  // namespace fdk

/* launch wrappers used by the host runtime */
extern "C" cudaError_t fdk_launch_geo_build(int nx, int ny, int nz, double h, double dq, double df, double z0r,
                                            const double *ysin, double *zrow, double *node, double *cell,
                                            cudaStream_t stream)
{
    fdk::fd_geo_build<<<152, 256, 0, stream>>>(nx, ny, nz, h, dq, df, z0r, ysin, zrow, node, cell);
    return cudaGetLastError();
}

/* shared memory per CTA that the dynamic part must leave: fd_solve's static shared memory, rounded
 * up to 1 KB */
static size_t dyn_smem_limit_margin()
{
    static size_t margin = 0;
    if (!margin) {
        cudaFuncAttributes a;
        margin = cudaFuncGetAttributes(&a, fdk::fd_solve) == cudaSuccess ? ((a.sharedSizeBytes + 1023) & ~(size_t)1023)
                                                                          : 4096;
    }
    return margin;
}

/* Launch shape of a batch: dynamic shared memory for the warp areas and the larger of the sweep-graph tables
 * (extents up to lmax, imax instances; 0: no station has a sweep graph) and, where stations walk their faces one at
 * a time, the largest such face's dependency bytes (max_face_pad points; left to global memory when they do not
 * fit).  Sets the kernel's shared-memory limit.  Host calls only (no stream work): done once per batch, outside any
 * capture. */
extern "C" cudaError_t fdk_solve_config(long long max_face_pad, int lmax, int imax, long long *bytes_out)
{
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const long long room = optin - (long long)dyn_smem_limit_margin();
    const long long base = (long long)fdk::kSmemBase;
    const long long graph = imax > 0 ? fdk::graph_smem_bytes(lmax, imax) : 0;
    const long long dagb = 2 * max_face_pad > graph ? 2 * max_face_pad : graph;
    const long long bytes = base + dagb <= room ? base + dagb : (base + graph <= room ? base + graph : base);
    /* the attribute is an upper bound shared by every launch of the kernel (a serving session may
     * launch it from another thread): always the largest */
    const cudaError_t e = cudaFuncSetAttribute(fdk::fd_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
    if (e != cudaSuccess) return e;
    *bytes_out = bytes;
    return cudaSuccess;
}

/* One launch of a configured batch: queues the kernel only (capturable in a CUDA graph). */
extern "C" cudaError_t fdk_solve_launch(const fd_station_dev *stations, int nst, long long bytes, int lmax, int imax,
                                        cudaStream_t stream)
{
    if (nst <= 0) return cudaSuccess;
    fdk::fd_solve<<<nst, FD_BLOCK, (size_t)bytes, stream>>>(stations, nst, (int)(bytes - fdk::kSmemBase), lmax, imax,
                                                           nullptr, 0);
    return cudaGetLastError();
}

extern "C" cudaError_t fdk_launch_solve(const fd_station_dev *stations, int nst, long long max_face_pad, int lmax,
                                        int imax, cudaStream_t stream)
{
    if (nst <= 0) return cudaSuccess;
    long long bytes = 0;
    const cudaError_t e = fdk_solve_config(max_face_pad, lmax, imax, &bytes);
    return e != cudaSuccess ? e : fdk_solve_launch(stations, nst, bytes, lmax, imax, stream);
}

/* The long-running grid of a serving session: nctas CTAs (one per SM), numbered cta_id0 onward in
 * q->exitf, with the largest dynamic shared memory a CTA can have (every request then finds the
 * sweep-graph tables and, when they fit, its face's dependency bytes in shared memory). */
extern "C" cudaError_t fdk_launch_serve(const fd_serve_queue *q, int nctas, int cta_id0, cudaStream_t stream)
{
    if (nctas <= 0) return cudaSuccess;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const long long bytes = optin - (long long)dyn_smem_limit_margin();
    const long long base = (long long)fdk::kSmemBase;
    if (bytes - base < fdk::graph_smem_bytes(FD_LMAX, FD_IMAX)) return cudaErrorInvalidConfiguration;
    /* the same bound as every other launch of the kernel */
    cudaError_t e = cudaFuncSetAttribute(fdk::fd_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    fdk::fd_solve<<<nctas, FD_BLOCK, (size_t)bytes, stream>>>(nullptr, 0, (int)(bytes - base), FD_LMAX, FD_IMAX, q, cta_id0);
    return cudaGetLastError();
}

/* dynamic shared memory a launch of fd_solve needs in the serving loop */
extern "C" long long fdk_serve_smem_bytes(void)
{
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return optin - (long long)dyn_smem_limit_margin();
}

#ifdef FD_SELFCHECK
/* the index-check record of FD_SELFCHECK builds: count, first site, first index; cleared after reading */
extern "C" cudaError_t fdk_selfcheck_read(unsigned long long *out)
{
    cudaError_t e = cudaMemcpyFromSymbol(out, fd_selfcheck_words, sizeof(unsigned long long) * 3);
    if (e == cudaSuccess) {
        const unsigned long long z[3] = {0, 0, 0};
        e = cudaMemcpyToSymbol(fd_selfcheck_words, z, sizeof z);
    }
    return e;
}
#endif

/* slowness = 1/velocity, float division as the reference does it (src/sphfd.c:689-690).  Bound by HBM: 16-byte
 * loads, kV2sBatch of them in flight per thread, where both arrays allow it (`wide`); else 4-byte loads, as many in
 * flight (the arrays may be one and the same, so that each load has to be written before the first store).
 * 401 x 401 x 161: 58.5 -> 34.3 us (6.0 TB/s) against a 4-byte load at a time; off a 16-byte boundary 62.1 -> 45.7. */
constexpr int kV2sBatch = 4, kV2sBlock = 256;

__global__ void __launch_bounds__(kV2sBlock) fd_v2s(const float *v, float *s, long long n, int wide)
{
    const long long first = (long long)blockIdx.x * kV2sBlock * kV2sBatch + threadIdx.x;
    if (!wide) {
        float a[kV2sBatch];
#pragma unroll
        for (int u = 0; u < kV2sBatch; u++)
            if (first + u * kV2sBlock < n) a[u] = v[first + u * kV2sBlock];
#pragma unroll
        for (int u = 0; u < kV2sBatch; u++)
            if (first + u * kV2sBlock < n) s[first + u * kV2sBlock] = 1.0f / a[u];
        return;
    }
    const long long n4 = n / 4;
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
    float4 *s4 = reinterpret_cast<float4 *>(s);
    float4 a[kV2sBatch];
#pragma unroll
    for (int u = 0; u < kV2sBatch; u++)
        if (first + u * kV2sBlock < n4) a[u] = v4[first + u * kV2sBlock];
#pragma unroll
    for (int u = 0; u < kV2sBatch; u++)
        if (first + u * kV2sBlock < n4)
            s4[first + u * kV2sBlock] = make_float4(1.0f / a[u].x, 1.0f / a[u].y, 1.0f / a[u].z, 1.0f / a[u].w);
    if (first < n - 4 * n4) s[4 * n4 + first] = 1.0f / v[4 * n4 + first];
}

extern "C" cudaError_t fdk_launch_v2s(const float *v, float *s, long long n, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    const int wide = ((reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(s)) & 15u) == 0;
    const long long per = (long long)kV2sBlock * kV2sBatch, items = wide ? (n + 3) / 4 : n;
    const long long blocks = (items + per - 1) / per;
    if (blocks > INT_MAX) return cudaErrorInvalidValue;
    fd_v2s<<<(int)blocks, kV2sBlock, 0, stream>>>(v, s, n, wide);
    return cudaGetLastError();
}

/* FP64 pipe rate probe: 8 independent fused multiply-add chains per thread, all SMs */
__global__ void fd_fp64_probe(double *out, int iters)
{
    double a0 = threadIdx.x * 1e-9 + 1.0, a1 = a0 + 1e-3, a2 = a0 + 2e-3, a3 = a0 + 3e-3;
    double a4 = a0 + 4e-3, a5 = a0 + 5e-3, a6 = a0 + 6e-3, a7 = a0 + 7e-3;
    const double m = 1.0000001, c = 1e-12;
    for (int i = 0; i < iters; i++) {
        a0 = __fma_rn(a0, m, c); a1 = __fma_rn(a1, m, c); a2 = __fma_rn(a2, m, c); a3 = __fma_rn(a3, m, c);
        a4 = __fma_rn(a4, m, c); a5 = __fma_rn(a5, m, c); a6 = __fma_rn(a6, m, c); a7 = __fma_rn(a7, m, c);
    }
    out[(long long)blockIdx.x * blockDim.x + threadIdx.x] = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
}

extern "C" cudaError_t fdk_probe_fp64(double *scratch, int blocks, int threads, int iters, float *ms, cudaStream_t s)
{
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    fd_fp64_probe<<<blocks, threads, 0, s>>>(scratch, iters);
    cudaEventRecord(e0, s);
    fd_fp64_probe<<<blocks, threads, 0, s>>>(scratch, iters);
    cudaEventRecord(e1, s);
    cudaError_t e = cudaEventSynchronize(e1);
    if (e == cudaSuccess) e = cudaEventElapsedTime(ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return e == cudaSuccess ? cudaGetLastError() : e;
}
