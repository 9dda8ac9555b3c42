// The V-th root of the Mul update's running product (mulprod_root, csrc/kernels.cuh) against doubles.
#include "kernels.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace {
__device__ __host__ unsigned mix(unsigned h)
{
    h *= 2654435761u;
    h ^= h >> 15;
    h *= 2246822519u;
    return h ^ h >> 13;
}
// mantissas of [0.5, 1) and exponents of -120 ... 120
__device__ __host__ float mantissa(int i) { return 0.5f + (float)(mix(i) & 0x7fffffu) * 5.9604644775390625e-8f; }
__device__ __host__ int exponent(int i) { return (int)(mix(~i) % 241) - 120; }
__global__ void k_root(int V, int n, float *out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = mvr::mulprod_root(make_float2(mantissa(i), (float)exponent(i)), V);
}
}  // namespace

// largest relative error over n values, or -1
extern "C" double root_error(int V, int n)
{
    float *d = nullptr;
    std::vector<float> h(n);
    if (cudaMalloc(&d, sizeof(float) * n) != cudaSuccess) return -1;
    k_root<<<512, 256>>>(V, n, d);
    const cudaError_t e = cudaMemcpy(h.data(), d, sizeof(float) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return -1;
    double m = 0.0;
    for (int i = 0; i < n; ++i) {
        const double r = std::pow((double)mantissa(i), 1.0 / V) * std::exp2((double)exponent(i) / V);
        m = std::max(m, std::fabs(h[i] / r - 1.0));
    }
    return m;
}
