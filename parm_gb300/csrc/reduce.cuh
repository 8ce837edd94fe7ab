// Block-wide FP64 sum or maximum in a fixed order, shared by the per-system
// reductions (integrate.cu) and the minimisers' fused sums (nlcg.cu).
#pragma once
#include <cuda_runtime.h>

namespace parm {

template <int NT>
__device__ __forceinline__ double block_reduce(double acc, bool is_max, double* sh) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_down_sync(0xFFFFFFFFu, acc, off);
        acc = is_max ? fmax(acc, o) : acc + o;
    }
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    double v = 0.0;
    if (threadIdx.x < 32) {
        v = threadIdx.x < NT / 32 ? sh[threadIdx.x] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_down_sync(0xFFFFFFFFu, v, off);
            v = is_max ? fmax(v, o) : v + o;
        }
    }
    __syncthreads();
    return v;   // valid in thread 0
}

constexpr int RED_THREADS = 256;

}  // namespace parm
