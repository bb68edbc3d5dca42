/* compares recip() with 1.f/t for every float it accepts; counts[0] differing, [1] accepted */
#include <cuda_runtime.h>

#include "fdgpu_recip.cuh"

__global__ void recip_kernel(unsigned long long *out)
{
    unsigned long long bad = 0, ok = 0;
    for (unsigned long long u = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; u < (1ull << 32);
         u += (unsigned long long)gridDim.x * blockDim.x) {
        const float t = __uint_as_float((unsigned)u);
        if (!recip_ok(t)) continue;
        ok++;
        bad += __float_as_uint(recip(t)) != __float_as_uint(1.f / t);
    }
    atomicAdd(&out[0], bad);
    atomicAdd(&out[1], ok);
}

extern "C" int recip_check(unsigned long long *counts)
{
    unsigned long long *out = nullptr;
    if (cudaMalloc(&out, 2 * sizeof *out) || cudaMemset(out, 0, 2 * sizeof *out)) return 1;
    recip_kernel<<<152 * 8, 256>>>(out);
    const cudaError_t e = cudaMemcpy(counts, out, 2 * sizeof *out, cudaMemcpyDeviceToHost);
    cudaFree(out);
    return e == cudaSuccess ? 0 : 2;
}
