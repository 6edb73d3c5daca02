// pic_spectral_dev.cuh -- arguments and helpers shared by the spectral solve's
// kernels (pic_spectral.cu, pic_spectral_small.cu, pic_spectral_mixed.cu).
#pragma once
#include <cuda_runtime.h>

#include "pic_adjoint_dev.cuh"
#include "pic_ensemble.cuh"
#include "pic_fft_dev.cuh"
#include "pic_field_dev.cuh"

namespace pic {

struct SpecArgs {
    unsigned long long *rho_fix;  // read by the forward rows, cleared by the columns
    float *rho;
    float2 *S;           // [nh][ny]: rows transformed along x
    float2 *Tx, *Ty;     // [nh][ny]: Ex~, Ey~ after the inverse along y
    float *ex, *ey;      // [ny][nx]
    const float2 *twx, *twy;
    int nx, ny, nh, lgx, lgy;
    long long mean_fix;
    float scale;
    float kx1, ky1, inv_eps0_n;
    int tmx, tmy;
    // adjoint solve (psi = S^T g): the two gradient planes in, their half
    // spectra in S and Sy, psi^ after the inverse along y in Tx; the inverse
    // rows take rows y ys and y ys + yo of Tx and Ty into ex and ey (ys = 1,
    // yo = 0 for the field; 2 and 1 for psi, two rows per transform)
    float *gx, *gy;  // cleared by the columns
    float2 *Sy;
    int ys, yo;
    int pairs, cols, rows;  // transforms (row pairs or rows), columns, rows per block
    int sa, sb, sc;         // buffer strides (float2) of the three kernels
    DevState *dev;
    // diagnostics folds of the step (0: none), by one block of the inverse rows
    double *hist;
    int hist_cap, adv;
    double fe_scale;
    // ensemble: blockIdx.y picks run first + blockIdx.y of this table, whose
    // grids sit at its offsets from the pointers above and whose constants
    // replace the ones above (nullptr: a single run)
    const EnsRun *runs;
    int first;
    int late;  // waits at its end (see pdl_wait): another group's kernel of this stage went before
};

// the arguments of this block's run
__device__ __forceinline__ SpecArgs block_args(const SpecArgs &P)
{
    SpecArgs A = P;
    if (P.runs) {
        const int r = P.first + (int)blockIdx.y;
        const EnsRun &R = P.runs[r];
        A.rho_fix = P.rho_fix + R.goff;
        A.rho = P.rho + R.goff;
        A.S = P.S + R.khoff;
        A.Tx = P.Tx + R.khoff;
        A.Ty = A.Tx + R.nk;
        A.ex = P.ex + 2 * R.goff;
        A.ey = A.ex + R.ncp;
        A.mean_fix = R.mean_fix;
        A.scale = R.rho_scale;
        A.kx1 = R.kx1;
        A.ky1 = R.ky1;
        A.inv_eps0_n = R.inv_eps0_n;
        A.dev = P.dev + r;
        A.hist = P.hist + (size_t)r * 6 * P.hist_cap;
        A.fe_scale = R.fe_scale;
    }
    return A;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) { return warp_sum_u64(v); }
__device__ __forceinline__ double warp_sum(double v) { return warp_sum_d(v); }

// Sum of v over the block, valid in thread 0.  Blocks of the small grids have
// fewer than 32 threads (a partial warp, where full-warp shuffles are not
// defined): their threads add through shared memory.  part: 32 entries.
template <class T>
__device__ __forceinline__ T block_sum(T v, T *part)
{
    if (blockDim.x >= 32) {
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    } else {
        part[threadIdx.x] = v;
    }
    __syncthreads();
    T s = 0;
    if (threadIdx.x == 0) {
        const int np = blockDim.x >= 32 ? (int)(blockDim.x >> 5) : (int)blockDim.x;
        for (int w = 0; w < np; ++w) s += part[w];
    }
    return s;
}

// ---- the solve in one cluster (pic_spectral_small.cu)
constexpr int CL = 8;  // blocks per cluster (the portable maximum)

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// (the built-in barriers, not inline asm: the compiler must not move threads of
// a warp that took different branches to separate copies of one)
__device__ __forceinline__ void cluster_arrive() { __cluster_barrier_arrive(); }
__device__ __forceinline__ void cluster_wait() { __cluster_barrier_wait(); }
// the address of this block's `p` in block `rank` of the cluster
__device__ __forceinline__ unsigned remote(const void *p, unsigned rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(r)
        : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void put2(unsigned a, float2 v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void put4(unsigned a, float2 u, float2 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(u.x), "f"(u.y),
                 "f"(v.x), "f"(v.y)
                 : "memory");
}
__device__ __forceinline__ void put(unsigned a, unsigned long long v)
{
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// The kernels of a solve and their launch shapes: three, or one (kernel[1] null).
struct SpecLaunch {
    SpecArgs A;
    const void *kernel[3];
    dim3 grid[3], block[3];
    size_t smem[3];
};

// the field solve's arguments on a handle (e: nullptr, or planes to write
// instead of the handle's)
void spectral_args(pic_handle *h, int adv, float *e, SpecArgs &A);
// pic_spectral_small.cu: the whole field solve of `batch` runs in one kernel, for
// the sides it takes (leaves L alone otherwise)
bool plan_small(SpecLaunch &L, int lgx, int lgy, int batch);

}  // namespace pic
