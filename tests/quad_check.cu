/*
 * quad_check.cu — test harness: the stencils as four lanes evaluate them (eval_corners_quad,
 * eval_edges_quad, which the solver runs for few items) against the one-lane forms (eval_3d, eval_ne and
 * eval_2d with the causality selection), bit for bit, on random and near-degenerate inputs over a real geometry.
 *
 * Built by tests/test_gpu_quad.py with nvcc into a temporary directory; it includes the kernel
 * translation unit so that it uses the same tables, descriptors and evaluators as the solver.
 */
#include "../fdtomoc_gb300/csrc/fdgpu_kernels.cu"

#include <cmath>
#include <vector>

namespace {
using namespace fdk;

__device__ __forceinline__ float unif(unsigned long long &s)
{
    s += 0x9e3779b97f4a7c15ull;
    unsigned long long x = (s ^ (s >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    x ^= x >> 31;
    return (float)((x >> 40) & 0xffffff) * (1.0f / 16777216.0f);
}

/* A block is a warp.  Per round: a face, a kind of trial (0 corner, 1 new edge, 2 two-dimensional), 1 to 8 items of different
 * slots, a slot a lane.  out: per kind, items, differing items, items with a root. */
__global__ void quad_kernel(fd_geo_dev g, unsigned long long seed, int rounds, unsigned long long *out)
{
    __shared__ WarpSmem ws;
    __shared__ TrialDesc dsc[FDN_NTRIAL];
    __shared__ fd_station_dev sd;
    const int lane = threadIdx.x;
    if (lane == 0) sd.g = g;
    unsigned long long s = seed + (blockIdx.x * 32ull + lane) * 0x2545f4914f6cdd1dull;
    unsigned long long common = seed ^ (blockIdx.x * 0x9e3779b97f4a7c15ull);   /* the same in all lanes */
    for (int r = 0; r < rounds; r++) {
        const int F = (int)(unif(common) * 6.f) % 6, kind = (int)(unif(common) * 3.f) % 3, n = 1 + (int)(unif(common) * 8.f) % 8;
        const int k0 = kind == 0 ? 0 : kind == 1 ? TK_NE0 : TK_2D0, kn = kind == 2 ? 8 : 4;
        __syncwarp();
        if (lane < FDN_NTRIAL) dsc[lane] = c_desc[F * FDN_NTRIAL + lane];
        ws.z[lane] = 1 + (int)(unif(s) * (float)(g.nz - 3));
        ws.y[lane] = 1 + (int)(unif(s) * (float)(g.ny - 3));
        const float base = unif(s) < 0.1f ? unif(s) * 0.05f : unif(s) * 80.f, slow = 0.1f + 0.25f * unif(s);
        const float size = slow * (unif(s) < 0.5f ? 1.f : 2.5f * unif(s)), jit = unif(s) < 0.3f ? 0.f : 0.05f * unif(s) * slow;
        const float gu = size * (2.f * unif(s) - 1.f), gv = size * (2.f * unif(s) - 1.f), gw = size * (2.f * unif(s) - 1.f);
        for (int nb = 0; nb < NB_N; nb++) {
            const int w = nb / 9, dv = (nb / 3) % 3 - 1, du = nb % 3 - 1;
            ws.t[lane][nb] = fmaxf(0.f, base + 0.5f * (gu * du + gv * dv + gw * w) + jit * (2.f * unif(s) - 1.f));
            ws.s[lane][nb] = slow * (1.f + 0.05f * (2.f * unif(s) - 1.f));
        }
        const bool none = unif(s) < 0.5f;   /* the inherited state: none, or near the times */
        ws.s0[lane] = none ? __int_as_float(0xff800000) : base + size * (unif(s) - 0.5f);
        ws.s4[lane] = none ? __int_as_float(0xff800000) : base + size * (unif(s) - 0.5f);
        const int shift = (int)(unif(common) * 32.f) % 32;
        if (lane < n) ws.items[lane] = (unsigned short)(((lane * 5 + shift) & 31) << 5 | (k0 + (int)(unif(s) * (float)kn) % kn));
        __syncwarp();
        if (kind == 0) eval_corners_quad(sd, dsc, ws, ws.items, n, lane);
        else eval_edges_quad(sd, dsc, ws, ws.items, n, lane);
        if (lane < n) {
            const int slot = ws.items[lane] >> 5, K = ws.items[lane] & 31, z = ws.z[slot], y = ws.y[slot];
            const float *t = ws.t[slot], *sl = ws.s[slot];
            const TrialDesc &d = dsc[K];
            double v;
            if (kind == 0) {
                v = eval_3d(d, t, sl, g, z, y);
            } else if (kind == 1) {
                v = eval_ne(d, t, sl, g, z, y);
            } else {
                double x1, x2;
                eval_2d(d, t, sl, g, z, y, x1, x2);
                const float fl = fmaxf(fmaxf(fmaxf(t[d.slot[1]], t[d.slot[2]]), fmaxf(t[d.slot[3]], ws.s0[slot])), ws.s4[slot]);
                const double f = (double)fl;
                if (x1 != x1) v = 1.e11;
                else if (x1 < f) v = x2 < f ? 1.e11 : x2;
                else v = x2 < f ? x1 : (x2 < x1 ? x2 : x1);
            }
            atomicAdd(&out[3 * kind], 1ull);
            if (__double_as_longlong(v) != __double_as_longlong(ws.res[slot][K])) atomicAdd(&out[3 * kind + 1], 1ull);
            if (v < 1.e11) atomicAdd(&out[3 * kind + 2], 1ull);
        }
        __syncwarp();
    }
}

}  // namespace

extern "C" int quad_check(int nx, int ny, int nz, double h, double dq, double df, double z0r, double y0, int rounds,
                          unsigned long long seed, unsigned long long *counts)
{
    std::vector<double> ys(ny);
    for (int y = 0; y < ny; y++) ys[y] = std::sin(y0 + dq * (double)y);
    double *ysin = nullptr, *zrow = nullptr, *node = nullptr, *cell = nullptr;
    unsigned long long *out = nullptr;
    if (cudaMalloc(&ysin, sizeof(double) * ny) || cudaMalloc(&zrow, sizeof(double) * FD_Z_N * nz)
        || cudaMalloc(&node, sizeof(double) * FD_N_N * (size_t)nz * ny)
        || cudaMalloc(&cell, sizeof(double) * FD_C_N * (size_t)(nz - 1) * (ny - 1))
        || cudaMalloc(&out, 9 * sizeof(unsigned long long)))
        return 1;
    cudaMemcpy(ysin, ys.data(), sizeof(double) * ny, cudaMemcpyHostToDevice);
    cudaMemset(out, 0, 9 * sizeof(unsigned long long));
    fdk_launch_geo_build(nx, ny, nz, h, dq, df, z0r, ysin, zrow, node, cell, 0);
    fd_geo_dev g;
    g.nx = nx; g.ny = ny; g.nz = nz;
    g.h = h; g.inv_h = 1.0 / h; g.dq = dq; g.df = df; g.is_h = 1.0 / (h * h);
    g.zrow = zrow; g.ysin = ysin; g.node = node; g.cell = cell;
    quad_kernel<<<152 * 2, 32>>>(g, seed, rounds, out);
    const cudaError_t e = cudaMemcpy(counts, out, 9 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
    cudaFree(ysin); cudaFree(zrow); cudaFree(node); cudaFree(cell); cudaFree(out);
    return e == cudaSuccess ? 0 : 2;
}
