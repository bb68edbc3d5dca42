/* The correctly rounded single-precision reciprocal, without a branch, for t from 2^-64 up to 2^64: an
 * approximation good to one unit in the last place and one Newton step in fused operations, which rounds correctly
 * (Markstein 1990, IBM J. Res. Dev. 34(1)).  Equal to 1.f/t for every float of the range. */
#ifndef FDGPU_RECIP_CUH
#define FDGPU_RECIP_CUH

constexpr unsigned kRecipLow = 0x1f800000u, kRecipSpan = 0x40000000u;   /* the range, as bits */

__device__ __forceinline__ bool recip_ok(float t) { return __float_as_uint(t) - kRecipLow < kRecipSpan; }

__device__ __forceinline__ float recip(float t)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(t));
    return fmaf(fmaf(-t, y, 1.f), y, y);
}

#endif
