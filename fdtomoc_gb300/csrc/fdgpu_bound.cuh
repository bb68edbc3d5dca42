/*
 * fdgpu_bound.cuh — single-precision lower bounds of stencil values, used to skip FP64
 * evaluations that cannot lower a running minimum.
 *
 * Most 2-D (fdsph2d) trials that pass the causality-floor test still lose to the running minimum
 * by far more than single-precision rounding: on the 201x201x81 benchmark station, 29 of 30 million
 * lose by more than 1e-4 relative, and only about 50 thousand win.  The FP64 pipe of this GPU is
 * narrow, so each skipped evaluation saves about 70 FP64 operations.
 *
 * The bound is rigorous, not a heuristic.  The stencil solves (x/d02 + p)^2 + (x/d01 + q)^2 = g with
 * p = (t1 - t3)/d13 - t2/d02 and q = (t2 - t3)/d23 - t1/d01, and shifting every time by t3 leaves the same
 * equation for x - t3: with alpha = t1 - t3 and beta = t2 - t3 (each one float subtraction) all terms are of
 * the size of a step's time, so FP32 loses little, and one forward error analysis bounds it:
 *   - with P = |alpha|/d13 + |beta|/d02, Q likewise, B = 2 (P/d02 + Q/d01), C = P^2 + Q^2 + g: the FP32
 *     discriminant is within 4 eps (B^2 + 4 a C) of the exact one, eps = 2^-21 (table doubles enter
 *     truncated, 2^-23 each; every operation adds 2^-24); FB_E32 doubles that;
 *   - the FP64 path forms the discriminant from the unshifted times: with T the largest time and v the
 *     largest reciprocal it is within 1408 2^-53 T^2 v^4 of the exact one; FB_E64 is 20 times that;
 *   - FB_EY covers the quotient (reciprocal, product and square root within 2^-21 each) and FB_ET T the
 *     FP64 path's own rounding of x.
 * Table doubles enter through truncation toward zero to FP32.  A NaN or an
 * overflow anywhere makes the result NaN and the final comparison fail, so the caller evaluates the
 * trial in FP64.  (Error bounds carried along through every operation, the form this replaces, took 350
 * instructions a trial where this takes about 90.)
 *
 * The kernel translation unit is compiled with --fmad=false, so the FP32 value operations are
 * rounded one by one, as the bound assumes.
 */
#ifndef FDGPU_BOUND_CUH
#define FDGPU_BOUND_CUH

#include "fdgpu_trials.cuh"

namespace fdk {

#define FB_E32 3.814697265625e-06f        /* 2^-18 */
#define FB_E64 3.637978807091713e-12f     /* 2^-38 */
#define FB_EB 9.5367431640625e-07f        /* 2^-20 */
#define FB_EY 1.9073486328125e-06f        /* 2^-19 */
#define FB_ET 9.094947017729282e-13f      /* 2^-40 */

/* a positive double truncated to float; NaN outside float's normal range, which makes every later
 * comparison fail */
__device__ __forceinline__ float d2f_trunc(double x)
{
    const float f = __double2float_rz(x);
    return f >= 1.17549435e-38f && f < 3.40282347e38f ? f : __int_as_float(0x7fc00000);
}

/* truncated reciprocals of the two tabulated distances at (z,y) (see FD_N_INV32) */
__device__ __forceinline__ float2 inv32_at(const fd_geo_dev &g, int z, int y)
{
    return *reinterpret_cast<const float2 *>(node_row(g, z, y) + FD_N_INV32);
}

/* square root and reciprocal within 2^-22 (the hardware's approximations are within 2^-23) */
__device__ __forceinline__ float sqrt_fast(float x)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* Lower bound of the value fdsph2d returns for trial d (the stencil of eval_2d), given its causality
 * floor fl or any float below it.  The roots of a x^2 + b x + c
 * (a > 0) satisfy x2 <= x1 in FP64 as well, every operation there being monotone, and the value is
 * x2 when x2 >= floor, else x1 when x1 >= floor, else the rejection value 1e11.  So when x2 is
 * certainly below fl the value is at least min(x1, 1e11); otherwise it is at least x2.  A floor
 * below the true one (the stale pair left out) only weakens the first test. */
__device__ __forceinline__ float lower_2d(const TrialDesc &d, const float *t18, const float *s18, const fd_geo_dev &g,
                                          int z, int y, float fl)
{
    const float inv_h = d2f_trunc(g.inv_h);
    float iv[4];   /* reciprocals of d01 d02 d13 d23 */
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = inv32_at(g, z + d.ddz[j], y + d.ddy[j]);
        iv[j] = d.dcls[j] == CH_H ? inv_h : d.dcls[j] == CH_RDQ ? f.x : f.y;
    }
    const float t1 = t18[d.slot[1]], t2 = t18[d.slot[2]], t3 = t18[d.slot[3]];
    const float al = t1 - t3, be = t2 - t3;
    const float sum = ((s18[NB_POINT] + s18[d.slot[1]]) + s18[d.slot[2]]) + s18[d.slot[3]];
    const float gg = sum * sum * 0.25f;
    const float u = al * iv[2], v = be * iv[1], w = be * iv[3], x = al * iv[0];
    const float p = u - v, q = w - x;
    const float P = fabsf(u) + fabsf(v), Q = fabsf(w) + fabsf(x);
    const float b = 2.f * (p * iv[1] + q * iv[0]), B = 2.f * (P * iv[1] + Q * iv[0]);
    const float c = (p * p + q * q) - gg, C = (P * P + Q * Q) + gg;
    const float a = iv[0] * iv[0] + iv[1] * iv[1], a4 = 4.f * a;
    const float rad = b * b - a4 * c, R = B * B + a4 * C;
    const float T = fmaxf(fmaxf(t1, t2), t3);
    const float vm = fmaxf(fmaxf(iv[0], iv[1]), fmaxf(iv[2], iv[3])), z64 = T * (vm * vm);
    const float E = FB_E32 * R + FB_E64 * (z64 * z64);
    if (!(E < 1.e30f)) return __int_as_float(0x7fc00000);
    if (rad + E < 0.f) return 1.e10f;   /* the FP64 discriminant is negative: 1e11 */
    const float shi = sqrt_fast(rad + E) * 1.00000095367431640625f;
    const float slo = sqrt_fast(fmaxf(rad - E, 0.f)) * 0.99999904632568359375f;
    const float i2a = rcp_fast(2.f * a);
    const float m = ((fabsf(b) + shi) * FB_EY + B * FB_EB) * i2a * 1.001f + FB_ET * T;
    if (__fadd_ru(t3, (-b - slo) * i2a + m) < fl) return fminf(__fadd_rd(t3, (slo - b) * i2a - m), 1.e10f);
    return __fadd_rd(t3, (-b - shi) * i2a - m);
}

}  // namespace fdk

#endif
