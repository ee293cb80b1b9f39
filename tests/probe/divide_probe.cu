// Test-only probe of divide_pair (th_common.cuh): how many of the given
// dividend pairs and divisors give another bit pattern than __fdiv_rn.
#include "../../torchhull_gb300/csrc/th_common.cuh"

__global__ void compare(const float* a, const float* b, const float* d, long long n, unsigned long long* differ)
{
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    unsigned long long bad = 0;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        float x, y;
        th::divide_pair(a[i], b[i], d[i], x, y);
        bad += __float_as_uint(x) != __float_as_uint(__fdiv_rn(a[i], d[i]));
        bad += __float_as_uint(y) != __float_as_uint(__fdiv_rn(b[i], d[i]));
    }
    if (bad)
        atomicAdd(differ, bad);
}

extern "C" int divide_probe(const float* a, const float* b, const float* d, long long n, unsigned long long* differ)
{
    compare<<<608, 256>>>(a, b, d, n, differ);
    return cudaDeviceSynchronize();
}
