// div_known against the general division, for test_gpu_div_known.py:
// differing results among n operands.
#include "pic_div_dev.cuh"

namespace {
__device__ bool differ(double a, double b, double y) { return pic::div_known(a, b, y) != __ddiv_rn(a, b); }

__global__ void given(const double *a, long long n, double b, double y, unsigned long long *bad)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && differ(a[i], b, y)) atomicAdd(bad, 1ull);
}

// random mantissas, exponents from -lo to hi
__global__ void drawn(unsigned long long seed, long long n, int lo, int hi, double b, double y, unsigned long long *bad)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);  // splitmix64
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const int e = -lo + (int)(z % (unsigned)(lo + hi + 1));
    const double m = 1.0 + (double)(z >> 12) * 0x1p-52;
    if (differ(ldexp((z & 2048) ? -m : m, e), b, y)) atomicAdd(bad, 1ull);
}
}  // namespace

extern "C" long long div_given(const double *a, long long n, double b)
{
    double *d = nullptr;
    unsigned long long *bad = nullptr, out = ~0ull;
    if (cudaMalloc(&d, n * 8) != cudaSuccess || cudaMalloc(&bad, 8) != cudaSuccess) return -1;
    cudaMemcpy(d, a, n * 8, cudaMemcpyHostToDevice);
    cudaMemset(bad, 0, 8);
    given<<<(unsigned)((n + 255) / 256), 256>>>(d, n, b, 1.0 / b, bad);
    const cudaError_t e = cudaMemcpy(&out, bad, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(bad);
    return e == cudaSuccess ? (long long)out : -1;
}

extern "C" long long div_drawn(unsigned long long seed, long long n, int lo, int hi, double b)
{
    unsigned long long *bad = nullptr, out = ~0ull;
    if (cudaMalloc(&bad, 8) != cudaSuccess) return -1;
    cudaMemset(bad, 0, 8);
    drawn<<<(unsigned)((n + 255) / 256), 256>>>(seed, n, lo, hi, b, 1.0 / b, bad);
    const cudaError_t e = cudaMemcpy(&out, bad, 8, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return e == cudaSuccess ? (long long)out : -1;
}
