// The adjoint's kick (adj_kick_block) on arrays of the caller's, for
// test_gpu_kick_block.py: one grid, no field, one anchor per block of `chunk`
// particles.  Scatter planes out (nx ny floats each).
#include <cstring>

#include "pic_adjoint_dev.cuh"

namespace {
__global__ void __launch_bounds__(256, 3)
kick(pic::KickArgs A, pic::KickGeo K, const int *anchor, int chunk, long long n)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const long long base = (long long)blockIdx.x * chunk;
    pic::adj_kick_block<false>(A, K, smem, base, min(base + (long long)chunk, n), anchor[blockIdx.x]);
}
}  // namespace

// n: a multiple of 4; returns a cudaError_t
extern "C" int kick_scatter(int nx, int ny, int tw, int th, int halo, long long n, int chunk,
                            const int *anchor, const int *cell, const float *ox, const float *oy,
                            const float *avx, const float *avy, float *gx, float *gy)
{
    const size_t nc = (size_t)nx * ny, bytes = (size_t)n * 4;
    const int blocks = (int)((n + chunk - 1) / chunk);
    float *p = nullptr;
    int *anc = nullptr;
    if (cudaMalloc(&p, 7 * bytes + 4 * nc * 4) != cudaSuccess) return (int)cudaGetLastError();
    if (cudaMalloc(&anc, blocks * 4) != cudaSuccess) return (int)cudaGetLastError();
    float *f[7];
    for (int k = 0; k < 7; ++k) f[k] = p + k * n;
    float *const planes = p + 7 * n;  // gx, gy, ex, ey
    cudaMemset(p, 0, 7 * bytes + 4 * nc * 4);
    const void *src[7] = {cell, ox, oy, nullptr, nullptr, avx, avy};
    for (int k = 0; k < 7; ++k)
        if (src[k]) cudaMemcpy(f[k], src[k], bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(anc, anchor, blocks * 4, cudaMemcpyHostToDevice);
    pic::KickArgs A = {(const int32_t *)f[0], f[1], f[2], nullptr, nullptr, f[3], f[4], f[5], f[6]};
    pic::KickGeo K;
    memset(&K, 0, sizeof K);
    K.G.nx = nx;
    K.G.ny = ny;
    K.G.tw = tw;
    K.G.th = th;
    K.G.hx = K.G.hy = halo;
    K.G.wcx = 2 * tw + 2 * halo;
    K.G.wcy = th + 2 * halo;
    K.gx = planes;
    K.gy = planes + nc;
    K.G.ex = planes + 2 * nc;
    K.G.ey = planes + 3 * nc;
    K.muc = 1.f;
    K.inv_dx = K.inv_dy = 1.f;
    const size_t smem = pic::kick_bytes(K.G.wcx, K.G.wcy);
    cudaFuncSetAttribute(kick, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kick<<<blocks, 256, smem>>>(A, K, anc, chunk, n);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaMemcpy(gx, planes, nc * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(gy, planes + nc, nc * 4, cudaMemcpyDeviceToHost);
    cudaFree(p);
    cudaFree(anc);
    return (int)e;
}
