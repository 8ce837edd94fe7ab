// Test-only: the radius and the angle of the Langevin normals (noise.cuh) of
// given 53-bit variates, so that their special cases can be asked for by value.
// Built by the tests.
#include <cstdint>
#include <cuda_runtime.h>

#include "noise.cuh"

__global__ void k_noise_words(const parm::NoiseTable* t, const unsigned long long* v, double* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[3 * (size_t)i] = parm::noise_radius(t, v[i]);
    parm::noise_turn(t, v[i], out[3 * (size_t)i + 1], out[3 * (size_t)i + 2]);
}

// variates in host memory -> (radius, cos, sin) each; 0 on success
extern "C" int noise_words(const uint64_t* v, double* out, uint32_t n) {
    if (n == 0) return 0;
    const parm::NoiseTable table = parm::make_noise_table();
    char* buf = nullptr;
    if (cudaMalloc(&buf, sizeof(table) + 32 * (size_t)n) != cudaSuccess) return 1;
    auto* t = reinterpret_cast<parm::NoiseTable*>(buf);
    auto* words = reinterpret_cast<unsigned long long*>(t + 1);
    auto* res = reinterpret_cast<double*>(words + n);
    int rc = 0;
    if (cudaMemcpy(t, &table, sizeof(table), cudaMemcpyHostToDevice) != cudaSuccess) rc = 2;
    if (!rc && cudaMemcpy(words, v, 8 * (size_t)n, cudaMemcpyHostToDevice) != cudaSuccess) rc = 2;
    if (!rc) {
        k_noise_words<<<(n + 255) / 256, 256>>>(t, words, res, n);
        if (cudaGetLastError() != cudaSuccess) rc = 3;
    }
    if (!rc && cudaMemcpy(out, res, 24 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) rc = 4;
    cudaFree(buf);
    return rc;
}
