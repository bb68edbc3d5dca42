/*
 * fdgpu_c2f.cu — coarse-to-fine model interpolation on the device: FDtomoC's c2f (reference
 * src/c2f.c), which turns the inversion's coarse P and S velocity nodes into the fine model sphfd
 * reads.  Results are bit-identical to the reference's.
 *
 * The reference places the coarse nodes at float coordinates accumulated step by step (:265-287),
 * turns the coarse velocities into slowness (:545-548), and for every fine node (x, y, z) = (x0 + i h,
 * ...) rounded to float scans for the coarse cell that holds it and interpolates the slowness
 * trilinearly in float (find_vel, :673-727), writing back 1/slowness (:561-572).
 *
 * GPU form: the cell and fractional offset along each axis depend only on that axis's fine index, so
 * the host forms them once per axis with the reference's float operations (nx + ny + nz entries), a
 * first kernel forms the coarse slowness, and the main kernel walks columns of fine nodes, combines the
 * three axes' entries into the eight weights, in the reference's order, and writes the velocity.  The slowness 1/v of the reference is computed in double and stored as float; float
 * division gives the same value (a double has more than twice a float's precision plus two bits, so
 * rounding the double quotient to float is the correctly rounded float quotient).  The main kernel
 * writes 8 bytes per fine node (P and S) and reads a coarse model that stays in L2.
 */
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

#include "fdgpu.h"
#include "fdgpu_device.h"
#include "fdgpu_recip.cuh"

namespace {

struct Axis {
    int cell;    /* coarse cell index */
    float f;     /* (v - g[cell]) / (g[cell+1] - g[cell]) */
    float omf;   /* 1 - f */
};

__global__ void c2f_slowness(const float *v, float *s, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s[i] = 1.f / v[i];
}

/* What bounds this is instruction issue (71 % of its slots, a third of them for pairs, which take two), then the
 * HBM writes: eight products of weight and slowness, their sum and a reciprocal per value written.  A thread takes two (x, y) of the plane, kC2fBlock apart so that each store
 * of a warp is contiguous (the plane is, rows included), and walks up a part of z: the four weight products of
 * x and y are formed once, the coarse slownesses stay in registers until z enters the next coarse cell, where
 * the upper four become the lower four, and P and S share the eight weights.  The two nodes are the halves of a
 * register pair, on which one instruction acts (each half rounded by itself).
 * 401 x 401 x 161: 149 -> 61 us (3.4 TB/s) against a warp per row with every value's weights and slownesses
 * formed anew; 78 us with one node a thread in single registers, 76 with pairs and a division per value. */
constexpr int kC2fBlock = 128;
constexpr int kC2fZ = 24;   /* fine planes a thread walks at most; 16 take 3 % longer, 48 the same */

struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
/* the product alone: a multiplication and an addition of pairs become one fused operation in the compiler, a
 * fused operation that adds -0 (which changes no product) does not, as long as it cannot see the -0 */
__device__ __forceinline__ F2 mul2(F2 a, F2 b, unsigned long long minus_zeros)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(minus_zeros));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__global__ void __launch_bounds__(kC2fBlock) c2f_interp(const float *__restrict__ slow, const Axis *__restrict__ ax,
                                                        const Axis *__restrict__ ay, const Axis *__restrict__ az,
                                                        int nx, int nxy, int nz, int across, int walk, int nxc, int nxyc, int ncoarse,
                                                        float *__restrict__ out, unsigned long long minus_zeros)
{
    __shared__ float2 zg[kC2fZ], zf[kC2fZ];   /* weights of the planes below and above, for both halves */
    __shared__ int zcell[kC2fZ + 1];
    const int part = blockIdx.x / across, col = blockIdx.x - part * across;   /* a thin model has more parts than grid.y takes */
    const int k0 = part * walk, nk = min(walk, nz - k0);
    if (threadIdx.x < nk) {
        const Axis Z = az[k0 + threadIdx.x];
        zg[threadIdx.x] = make_float2(Z.omf, Z.omf);
        zf[threadIdx.x] = make_float2(Z.f, Z.f);
        zcell[threadIdx.x] = Z.cell;
    }
    if (threadIdx.x == nk) zcell[nk] = -1;
    __syncthreads();
    const int p = col * 2 * kC2fBlock + threadIdx.x;
    if (p >= nxy) return;
    const bool two = p + kC2fBlock < nxy;
    const int p2 = two ? p + kC2fBlock : p;
    const int j = p / nx, j2 = p2 / nx;
    const Axis X = ax[p - j * nx], X2 = ax[p2 - j2 * nx], Y = ay[j], Y2 = ay[j2];
    const F2 gg = pack2(X.omf * Y.omf, X2.omf * Y2.omf), fg = pack2(X.f * Y.omf, X2.f * Y2.omf);
    const F2 gf = pack2(X.omf * Y.f, X2.omf * Y2.f), ff = pack2(X.f * Y.f, X2.f * Y2.f);
    const float *sa = slow + nxc * Y.cell + X.cell, *sb = slow + nxc * Y2.cell + X2.cell;
    /* the cell's lower and upper corners at (x, y), (x+1, y), (x, y+1), (x+1, y+1); P, S */
    F2 lo[2][4], hi[2][4];
    auto plane = [&](int cz, F2 c[2][4]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float *a = sa + cz * nxyc + h * ncoarse, *b = sb + cz * nxyc + h * ncoarse;
            c[h][0] = pack2(a[0], b[0]);
            c[h][1] = pack2(a[1], b[1]);
            c[h][2] = pack2(a[nxc], b[nxc]);
            c[h][3] = pack2(a[nxc + 1], b[nxc + 1]);
        }
    };
    const long long nfine = (long long)nxy * nz;
    float *o = out + (long long)k0 * nxy + p;
    int k = 0, cell = zcell[0];
    plane(cell, lo);
    for (;;) {
        plane(cell + 1, hi);
        do {
            auto w = [&](F2 xy, const float2 &z) { return mul2(xy, pack2(z.x, z.y), minus_zeros); };
            const F2 w0 = w(gg, zg[k]), w1 = w(fg, zg[k]), w2 = w(gf, zg[k]), w3 = w(gg, zf[k]), w4 = w(ff, zg[k]);
            const F2 w5 = w(fg, zf[k]), w6 = w(gf, zf[k]), w7 = w(ff, zf[k]);
            float t[4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                F2 s = mul2(w0, lo[h][0], minus_zeros);
                s = add2(s, mul2(w1, lo[h][1], minus_zeros));
                s = add2(s, mul2(w2, lo[h][2], minus_zeros));
                s = add2(s, mul2(w3, hi[h][0], minus_zeros));
                s = add2(s, mul2(w4, lo[h][3], minus_zeros));
                s = add2(s, mul2(w5, hi[h][1], minus_zeros));
                s = add2(s, mul2(w6, hi[h][2], minus_zeros));
                s = add2(s, mul2(w7, hi[h][3], minus_zeros));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(t[2 * h]), "=f"(t[2 * h + 1]) : "l"(s.v));
            }
            /* without the divisions' own branches the four reciprocals run side by side */
            if (recip_ok(t[0]) && recip_ok(t[1]) && recip_ok(t[2]) && recip_ok(t[3])) {
#pragma unroll
                for (int q = 0; q < 4; q++) t[q] = recip(t[q]);
            } else {
#pragma unroll 1
                for (int q = 0; q < 4; q++) {
                    const float v = 1.f / t[0];
                    t[0] = t[1];
                    t[1] = t[2];
                    t[2] = t[3];
                    t[3] = v;
                }
            }
            o[0] = t[0];
            o[nfine] = t[2];
            if (two) {
                o[kC2fBlock] = t[1];
                o[nfine + kC2fBlock] = t[3];
            }
            o += nxy;
            k++;
        } while (zcell[k] == cell);
        if (k == nk) break;
        if (zcell[k] == cell + 1) {
#pragma unroll
            for (int q = 0; q < 8; q++) lo[q / 4][q % 4] = hi[q / 4][q % 4];
        } else {
            plane(zcell[k], lo);
        }
        cell = zcell[k];
    }
}

/* the per-axis entries: node coordinates accumulated as the reference does, fine positions rounded
 * to float, the first node past each position less one (kept inside), and the offset */
void axis_table(int nc, const int *ig, double o, double h, int nfine, std::vector<Axis> &out)
{
    std::vector<float> g(nc);
    g[0] = (float)o;
    for (int i = 1; i < nc; i++) g[i] = (float)(g[i - 1] + h * ig[i - 1]);
    out.resize(nfine);
    for (int i = 0; i < nfine; i++) {
        const float v = (float)(o + i * h);
        int c;
        for (c = 1; c < nc; c++)
            if (g[c] > v) break;
        if (c == nc) c--;
        c--;
        const float f = (v - g[c]) / (g[c + 1] - g[c]);
        out[i].cell = c;
        out[i].f = f;
        out[i].omf = 1.f - f;
    }
}

int kind_of(const void *p, int device, bool *on_device)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        *on_device = false;
        return FDGPU_OK;
    }
    if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) {
        if (a.device != device) return FDGPU_EINVAL;
        *on_device = true;
    } else {
        *on_device = false;
    }
    return FDGPU_OK;
}

}  // namespace

extern "C" int fdh_ctx_device(const fdgpu_ctx *ctx);
extern "C" void *fdh_ctx_stream(const fdgpu_ctx *ctx);
extern "C" int fdh_ctx_fail(fdgpu_ctx *ctx, int cuda_error, const char *what);

extern "C" int fdgpu_c2f_dims(const fdgpu_c2f_grid *g, int *nx, int *ny, int *nz)
{
    if (!g || !nx || !ny || !nz || g->nxc < 2 || g->nyc < 2 || g->nzc < 2 || !g->igridx || !g->igridy || !g->igridz)
        return FDGPU_EINVAL;
    long long x = 1, y = 1, z = 1;
    for (int i = 1; i < g->nxc; i++) { if (g->igridx[i - 1] < 1) return FDGPU_EINVAL; x += g->igridx[i - 1]; }
    for (int i = 1; i < g->nyc; i++) { if (g->igridy[i - 1] < 1) return FDGPU_EINVAL; y += g->igridy[i - 1]; }
    for (int i = 1; i < g->nzc; i++) { if (g->igridz[i - 1] < 1) return FDGPU_EINVAL; z += g->igridz[i - 1]; }
    if (x * y * z >= (1ll << 31) || (long long)g->nxc * g->nyc * g->nzc >= (1ll << 30)) return FDGPU_EINVAL;
    *nx = (int)x;
    *ny = (int)y;
    *nz = (int)z;
    return FDGPU_OK;
}

struct fdgpu_c2f_plan {
    fdgpu_ctx *ctx = nullptr;
    int device = 0;
    int nx = 0, ny = 0, nz = 0, nxc = 0, nyc = 0, nzc = 0;
    int sms = 1;
    char *mem = nullptr;   /* slowness (2 x coarse), axis tables */
    float *slow = nullptr;
    Axis *ax = nullptr, *ay = nullptr, *az = nullptr;
};

extern "C" int fdgpu_c2f_plan_create(fdgpu_ctx *ctx, const fdgpu_c2f_grid *g, fdgpu_c2f_plan **out)
{
    if (!ctx || !out) return FDGPU_EINVAL;
    *out = nullptr;
    int nx, ny, nz;
    int rc = fdgpu_c2f_dims(g, &nx, &ny, &nz);
    if (rc) return rc;
    if (!(g->h > 0)) return FDGPU_EINVAL;
    const int dev = fdh_ctx_device(ctx);
    FdDeviceScope dev_(dev);
    if (dev_.err) return FDGPU_ENODEV;
    std::vector<Axis> ax, ay, az;
    axis_table(g->nxc, g->igridx, g->x0, g->h, nx, ax);
    axis_table(g->nyc, g->igridy, g->y0, g->h, ny, ay);
    axis_table(g->nzc, g->igridz, g->z0, g->h, nz, az);
    auto *p = new (std::nothrow) fdgpu_c2f_plan;
    if (!p) return FDGPU_ENOMEM;
    p->ctx = ctx;
    p->device = dev;
    p->nx = nx; p->ny = ny; p->nz = nz;
    p->nxc = g->nxc; p->nyc = g->nyc; p->nzc = g->nzc;
    if (cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || p->sms < 1) p->sms = 1;
    const size_t nc2 = 2 * (size_t)g->nxc * g->nyc * g->nzc;
    const size_t o_x = (sizeof(float) * nc2 + 255) & ~(size_t)255;
    const size_t o_y = o_x + ((sizeof(Axis) * nx + 255) & ~(size_t)255);
    const size_t o_z = o_y + ((sizeof(Axis) * ny + 255) & ~(size_t)255);
    const size_t total = o_z + sizeof(Axis) * nz;
    cudaError_t e = cudaMalloc((void **)&p->mem, total);
    if (!e) e = cudaMemcpy(p->mem + o_x, ax.data(), sizeof(Axis) * nx, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(p->mem + o_y, ay.data(), sizeof(Axis) * ny, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(p->mem + o_z, az.data(), sizeof(Axis) * nz, cudaMemcpyHostToDevice);
    if (e) {
        rc = fdh_ctx_fail(ctx, (int)e, "c2f plan");
        if (p->mem) cudaFree(p->mem);
        delete p;
        return rc;
    }
    p->slow = reinterpret_cast<float *>(p->mem);
    p->ax = reinterpret_cast<Axis *>(p->mem + o_x);
    p->ay = reinterpret_cast<Axis *>(p->mem + o_y);
    p->az = reinterpret_cast<Axis *>(p->mem + o_z);
    *out = p;
    return FDGPU_OK;
}

extern "C" int fdgpu_c2f_run(fdgpu_c2f_plan *p, const float *d_coarse, float *d_fine, void *stream)
{
    if (!p || !d_coarse || !d_fine) return FDGPU_EINVAL;
    cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)fdh_ctx_stream(p->ctx);
    FdDeviceScope dev_(p->device);
    if (dev_.err) return FDGPU_ENODEV;
    const int nc2 = 2 * p->nxc * p->nyc * p->nzc;
    c2f_slowness<<<(nc2 + 255) / 256 < 1024 ? (nc2 + 255) / 256 : 1024, 256, 0, st>>>(d_coarse, p->slow, nc2);
    const int nxy = p->nx * p->ny;
    const int across = (nxy + 2 * kC2fBlock - 1) / (2 * kC2fBlock);
    /* a model too small for eight blocks an SM is split further along z, to one plane a thread: there the
     * walk's latency is what takes the time (28 x 64 x 27: 16.6 us a call with 24 planes, 8.4 with one) */
    int walk = kC2fZ;
    while (walk > 1 && (long long)across * ((p->nz + walk - 1) / walk) < 8ll * p->sms) walk /= 2;
    const int grid = across * ((p->nz + walk - 1) / walk);
    c2f_interp<<<grid, kC2fBlock, 0, st>>>(p->slow, p->ax, p->ay, p->az, p->nx, nxy, p->nz, across, walk, p->nxc, p->nxc * p->nyc,
                                             p->nxc * p->nyc * p->nzc, d_fine, 0x8000000080000000ull);
    const cudaError_t e = cudaGetLastError();
    return e ? fdh_ctx_fail(p->ctx, (int)e, "c2f launch") : FDGPU_OK;
}

extern "C" void fdgpu_c2f_plan_destroy(fdgpu_c2f_plan *p)
{
    if (!p) return;
    FdDeviceScope dev_(p->device);
    if (p->mem) {
        cudaDeviceSynchronize();
        cudaFree(p->mem);
    }
    delete p;
}

extern "C" int fdgpu_c2f(fdgpu_ctx *ctx, const fdgpu_c2f_grid *g, const float *coarse, float *fine, void *stream)
{
    if (!ctx || !coarse || !fine) return FDGPU_EINVAL;
    fdgpu_c2f_plan *p = nullptr;
    int rc = fdgpu_c2f_plan_create(ctx, g, &p);
    if (rc) return rc;
    cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)fdh_ctx_stream(ctx);
    bool cin = false, cout = false;
    const long long nxyz = (long long)p->nx * p->ny * p->nz;
    const size_t nc2 = 2 * (size_t)p->nxc * p->nyc * p->nzc;
    float *dc = nullptr, *df = nullptr;
    cudaError_t e = cudaSuccess;
    if (kind_of(coarse, p->device, &cin) || kind_of(fine, p->device, &cout)) {
        fdgpu_c2f_plan_destroy(p);
        return FDGPU_EINVAL;
    }
    if (!cin) {
        e = cudaMallocAsync((void **)&dc, sizeof(float) * nc2, st);
        if (!e) e = cudaMemcpyAsync(dc, coarse, sizeof(float) * nc2, cudaMemcpyHostToDevice, st);
    }
    if (!e && !cout) e = cudaMallocAsync((void **)&df, sizeof(float) * 2 * (size_t)nxyz, st);
    if (!e) rc = fdgpu_c2f_run(p, cin ? coarse : dc, cout ? fine : df, st);
    if (!e && !rc && !cout) e = cudaMemcpyAsync(fine, df, sizeof(float) * 2 * (size_t)nxyz, cudaMemcpyDeviceToHost, st);
    if (dc) cudaFreeAsync(dc, st);
    if (df) cudaFreeAsync(df, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (!e) e = e2;
    if (e && !rc) rc = fdh_ctx_fail(ctx, (int)e, "c2f");
    fdgpu_c2f_plan_destroy(p);
    return rc;
}
