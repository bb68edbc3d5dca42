/*
 * fdgpu_eval.cuh — evaluation of one face point on the GPU, bit-identical to the reference.
 *
 * The reference's face-point body (TOP: src/sphfd.c:1034-1761, the other faces mirrored) runs 22
 * trial stencils in a fixed order and keeps the minimum.  The sequence comes from fd_face_table.h.
 * The arithmetic keeps the reference's FP64 operation order exactly; what changes is how each
 * operation is obtained:
 *
 *   - geometry-only subexpressions (products of radius, sin(colatitude), angular steps, the
 *     fdsph3d coefficients, the quadratics' 'a') come from tables built with the reference's own
 *     formula, so they are the same doubles the reference computes;
 *   - x / d for a geometric divisor d is RN(x/d) computed from the tabulated RN(1/d) with two
 *     fused-multiply-add corrections (Markstein's theorem; 5 FP64 ops instead of ~17 for a
 *     generic division on this part);
 *   - a stencil whose causality floor (the largest time it reads, which its accepted root can
 *     never be below) is already >= the running minimum is not evaluated: it cannot lower the
 *     minimum, and its only side effect, the stale (t0,t4) state, is still applied.
 *
 * The kernel translation unit is compiled with --fmad=false: no multiply-add is contracted except
 * the explicit __fma_rn corrections of the division, whose results are exact by construction.
 */
#ifndef FDGPU_EVAL_CUH
#define FDGPU_EVAL_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "fd_face_table.h"
#include "fdgpu_check.cuh"
#include "fdgpu_layout.h"

namespace fdk {

/* ---------------------------------------------------------------------------------------------- */
/* exact helpers                                                                                   */

/* Conversions, comparisons and products by powers of two are FP64 instructions, although each occupies the FP64 unit
 * for 64 cycles: the solver waits for instructions to arrive from the caches in half of its cycles, so
 * that sequences of four to twelve integer instructions in their place cost more (400 windows of 25 to 61: 186 ms
 * with such sequences, 172 without; one of 27x20x21: 4.78 and 4.69). */

__device__ __forceinline__ double f2d(float f) { return (double)f; }
__device__ __forceinline__ bool lt(double a, double b) { return a < b; }

/* RN(x / d) given inv = RN(1/d): q = RN(x*inv) then two exact-residual corrections.  Zero x keeps
 * its sign, as a true division would. */
__device__ __forceinline__ double div_rn(double x, double d, double inv)
{
    const double q0 = __dmul_rn(x, inv);
    double e = __fma_rn(-d, q0, x);
    const double q = __fma_rn(e, inv, q0);
    e = __fma_rn(-d, q, x);
    const double r = __fma_rn(e, inv, q);
    return (__double_as_longlong(x) << 1) == 0 ? q0 : r;
}

/* ---------------------------------------------------------------------------------------------- */
/* compile-time face geometry                                                                      */

template <int F>
struct FaceT {
    static constexpr int AU = fd_face_frame[F].axis_u;
    static constexpr int AV = fd_face_frame[F].axis_v;
    static constexpr int AN = fd_face_frame[F].axis_n;
    static constexpr int IN = fd_face_frame[F].inner;
    static constexpr int HW = fd_face_frame[F].headw;
    /* offset of node (du,dv,w) along grid axis a (0 x, 1 y, 2 z) */
    __host__ __device__ static constexpr int off(int a, fdn_node n) { return a == AU ? n.du : a == AV ? n.dv : n.w * IN; }
};

__device__ __forceinline__ const double *node_row(const fd_geo_dev &g, int z, int y)
{
    if (!FD_OK(z, g.nz, 1) || !FD_OK(y, g.ny, 2)) { z = 0; y = 0; }
    return g.node + (long long)(z * g.ny + y) * FD_N_N;   /* a face has at most 2^30 points */
}

/* canonical distance products of the new-edge / 2-D / new-face stencils */
enum { CH_H = 0, CH_RDQ = 1, CH_RSDF = 2 };
__host__ __device__ constexpr int chain_class(fdn_chain c)
{
    return c.n == 1 ? CH_H : c.n == 2 ? CH_RDQ : CH_RSDF;
}

/* roots of a x^2 + b x + c = 0 (rad = b*b - 4ac already formed), with the reference's
 * causality test against floor tmx; tie rule of fdsph3d (x1 preferred only if strictly smaller). */
__device__ __forceinline__ double roots_3d(double b, double rad, double twoa, double i2a, double tmx)
{
    if (!(rad >= 0.)) return 1.e11;
    const double sq = __dsqrt_rn(rad);
    const double x1 = div_rn(-b + sq, twoa, i2a);
    const double x2 = div_rn(-b - sq, twoa, i2a);
    const bool bad1 = x1 < tmx, bad2 = x2 < tmx;
    if (bad1) return bad2 ? 1.e11 : x2;
    if (bad2) return x1;
    return x1 < x2 ? x1 : x2;
}

/* same, with the tie rule of fdsphne / fdsph2d (x2 preferred only if strictly smaller) */
__device__ __forceinline__ double roots_2(double b, double rad, double twoa, double i2a, double tmx)
{
    if (!(rad >= 0.)) return 1.e11;
    const double sq = __dsqrt_rn(rad);
    const double x1 = div_rn(-b + sq, twoa, i2a);
    const double x2 = div_rn(-b - sq, twoa, i2a);
    const bool bad1 = x1 < tmx, bad2 = x2 < tmx;
    if (bad1) return bad2 ? 1.e11 : x2;
    if (bad2) return x1;
    return x2 < x1 ? x2 : x1;
}

}  // namespace fdk

#endif
