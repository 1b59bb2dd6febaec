// cnn_math.cuh — device functions shared by the closure network's FP32 and tensor-core training kernels.
#pragma once
#include <cuda_runtime.h>

namespace dns2d {
namespace cnn {

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z)
{
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// Column sums of G partials of 32 columns, `stride` floats apart: 32 threads groups of 8 lanes (a lane 4
// columns) take g = group, group + 32, ..., and lane i of the first warp returns column i's sum of the 32
// groups in order: FP64 throughout, a fixed order.  256 threads.
__device__ __forceinline__ double sum_partials(const float *__restrict__ part, int G, size_t stride)
{
    __shared__ double red[32][33];
    const int q = threadIdx.x & 7, grp = threadIdx.x >> 3;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int g = grp; g < G; g += 32) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(part + g * stride) + q);
        s[0] += (double)v.x;
        s[1] += (double)v.y;
        s[2] += (double)v.z;
        s[3] += (double)v.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) red[grp][4 * q + i] = s[i];
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32)
        for (int i = 0; i < 32; ++i) t += red[i][threadIdx.x];
    return t;
}

}  // namespace cnn
}  // namespace dns2d
