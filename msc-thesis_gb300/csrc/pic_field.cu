// pic_field.cu -- the grid side of the step: fixed-point density to float,
// the k-space Poisson kernel, and per-step diagnostics bookkeeping.
//
// Replaces (reference paths inside taylorj5/msc-thesis,
// thesisCode/collisionless/double/src/):
//   fourier.cc:15-126 fftPoissonSolver   -> convert + cuFFT R2C + kspace + cuFFT C2R
//   grid.cc:85-96     computeElectricField (the field comes from E^ = -i k phi^
//                                           in the same k-space kernel)
// with physical conventions: k = 2 pi m / L, phi^ = rho^ / (eps0 k^2), the
// zero mode removed (immobile neutralising background) and one 1/N.
#include <cuda_runtime.h>

#include "pic_field_dev.cuh"

namespace pic {

// rho = (rho_fix - mean) * scale, sum(rho_fix) -> dev->q; rho_fix is cleared
// by the k-space kernel.  The background is removed in exact integer
// arithmetic before the single rounding to float, so small perturbations of a
// large mean keep their relative precision.  Two cells per thread per
// iteration (16-byte loads, 8-byte stores; n is even).
__global__ void __launch_bounds__(256)
convert_kernel(const unsigned long long *rho_fix, float *__restrict__ rho, long long n, long long mean_fix,
               float scale, DevState *dev)
{
    __shared__ unsigned long long s_part[8];
    pdl_wait();
    pdl_trigger();
    unsigned long long qs = 0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long n2 = n >> 1;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(rho_fix)[i];
        qs += v.x + v.y;
        reinterpret_cast<float2 *>(rho)[i] =
            make_float2(fixed_to_float(v.x, mean_fix, scale), fixed_to_float(v.y, mean_fix, scale));
    }
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long v = rho_fix[n - 1];
        qs += v;
        rho[n - 1] = fixed_to_float(v, mean_fix, scale);
    }
    qs = warp_sum_u64(qs);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = qs;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
        atomicAdd(&dev->q[acc_slot()], t);
    }
}

struct KspaceArgs {
    const float2 *rhohat;
    float2 *ehat;    // [2][ny][nh] (E mode) or phi^ (phi mode)
    int nx, ny, nh;
    float kx1, ky1;  // 2 pi / Lx, 2 pi / Ly
    float inv_eps0_n;  // 1 / (eps0 nx ny): folds the C2R normalisation in
    int phi_mode;
    int tmx, tmy;      // tracked mode (tmx < 0: none)
    DevState *dev;
    unsigned long long *rho_fix;  // cleared here (already converted)
    double *hist;
    int hist_cap, adv;            // diagnostics folds of the step (0: none)
    double fe_scale;
};

// Blocks walk rows of the half spectrum, threads the modes of a row.  In E
// mode the kernel also clears the fixed-point density for the next deposit
// and its last block folds the step's diagnostics: launches of their own
// before (a memset and advance_kernel; 250 x 180 x 23 per cell with the
// chain's dependent launches: 56.3 to 55.6 us a step).
__global__ void __launch_bounds__(256) kspace_kernel(KspaceArgs A)
{
    __shared__ double s_part[8];
    __shared__ bool s_last;
    pdl_wait();
    pdl_trigger();
    if (!A.phi_mode) {
        const long long n = (long long)A.nx * A.ny, stride = (long long)gridDim.x * blockDim.x;
        const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        for (long long i = t0; i < n >> 1; i += stride)
            reinterpret_cast<ulonglong2 *>(A.rho_fix)[i] = make_ulonglong2(0ull, 0ull);
        if ((n & 1) && t0 == 0) A.rho_fix[n - 1] = 0ull;
    }
    const long long total = (long long)A.ny * A.nh;
    float fe = 0.f;
    for (int my = blockIdx.x; my < A.ny; my += gridDim.x)
    for (int mx = threadIdx.x; mx < A.nh; mx += blockDim.x) {
        const long long idx = (long long)my * A.nh + mx;
        const float2 r = A.rhohat[idx];
        const KMode K = kspace_mode(r, mx, my, A.nx, A.ny, A.kx1, A.ky1, A.inv_eps0_n, idx == 0);
        if (mx == A.tmx && my == A.tmy)
            A.dev->mode_amp = sqrt((double)r.x * r.x + (double)r.y * r.y) / ((double)A.nx * A.ny);
        if (A.phi_mode) {
            A.ehat[idx] = K.ph;
            continue;
        }
        A.ehat[idx] = K.ex;
        A.ehat[total + idx] = K.ey;
        fe += K.fe;
    }
    if (A.phi_mode) return;
    double d = warp_sum_d((double)fe);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
        atomicAdd(&A.dev->fe[acc_slot()], t);
        if (A.adv) {
            __threadfence();  // this block's sums before its ticket
            s_last = atomicInc(&A.dev->ticket, gridDim.x - 1) == gridDim.x - 1;
        }
    }
    if (!A.adv) return;
    __syncthreads();
    if (s_last && threadIdx.x < 32) {
        __threadfence();
        advance_state(A.dev, A.hist, A.hist_cap, A.adv, A.fe_scale, 32);
    }
}

// diagnostics fold of one handle (one warp)
__global__ void advance_kernel(DevState *d, double *hist, int cap, int kind, double fe_scale)
{
    pdl_wait();
    pdl_trigger();
    advance_state(d, hist, cap, kind, fe_scale, 32);
}

pic_status launch_convert(pic_handle *h)
{
    const Geometry &g = h->g;
    const long long n = (long long)g.nx * g.ny;
    float scale = (float)(h->q_unit / (4294967296.0 * g.dx * g.dy));
    long long nn = n;
    void *args[] = {&h->rho_fix, &h->rho, &nn, &h->mean_fix, &scale, &h->dev};
    return launch_dependent((const void *)convert_kernel, grid_for((n + 1) / 2, 256), 256, 0,
                            h->stream, args);
}

// sum_n |E_n|^2 = N sum_k |E'^_k|^2 with E' the 1/N-scaled spectrum
static double fe_scale_of(const pic_handle *h)
{
    const Geometry &g = h->g;
    return 0.5 * h->cfg.eps0 * g.dx * g.dy * (double)g.nx * (double)g.ny;
}

pic_status launch_kspace(pic_handle *h, bool phi_only, float2 *phihat, int adv)
{
    const Geometry &g = h->g;
    KspaceArgs A;
    A.rhohat = h->rhohat;
    A.ehat = phi_only ? phihat : h->ehat;
    A.nx = g.nx;
    A.ny = g.ny;
    A.nh = g.nh;
    A.kx1 = (float)(2.0 * 3.14159265358979323846 / g.Lx);
    A.ky1 = (float)(2.0 * 3.14159265358979323846 / g.Ly);
    A.inv_eps0_n = (float)(1.0 / (h->cfg.eps0 * (double)g.nx * (double)g.ny));
    A.phi_mode = phi_only ? 1 : 0;
    A.tmx = phi_only ? -1 : h->track_mx;
    A.tmy = phi_only ? -1 : h->track_my;
    A.dev = h->dev;
    A.rho_fix = h->rho_fix;
    A.hist = h->hist;
    A.hist_cap = h->hist_cap;
    A.adv = phi_only ? 0 : adv;
    A.fe_scale = fe_scale_of(h);
    void *args[] = {&A};
    return launch_dependent((const void *)kspace_kernel, grid_for((long long)g.ny * 256, 256), 256,
                            0, h->stream, args);
}

pic_status launch_advance(pic_handle *h, int kind)
{
    double fe_scale = fe_scale_of(h);
    void *args[] = {&h->dev, &h->hist, &h->hist_cap, &kind, &fe_scale};
    return launch_dependent((const void *)advance_kernel, 1, 32, 0, h->stream, args);
}

}  // namespace pic
