// pic_compat.cu -- the reference's step, with its CPU conventions, in FP64 on
// the GPU: the drop-in for picFloatGpu.
//
// Follows, operation for operation where the GPU allows (reference paths in
// taylorj5/msc-thesis, thesisCode/collisionless/double/):
//   src/grid.cc:46-76      chargeAssignment: CIC weights to the opposite corner
//                          nodes, written at ghost-padded index (1+cx, 1+cy),
//                          q*w per node, then the periodic ghost copy
//   src/fourier.cc:15-126  fftPoissonSolver: k = 2 pi m, the second index
//                          mapped with `2*j < nyh` (so j >= nyh/2 maps to j-ny),
//                          phi^ = -rho^/k^2, normalised twice by 1/(nx ny)
//   src/grid.cc:85-96      computeElectricField: central differences, Ex along
//                          the second index, Ey along the first, interior only
//   src/particle.cc:37-106 forceCalculation (E read at (cx, cy) without the
//                          ghost offset) and the lagged kick-drift-kick
//                          positionUpdate with forceOld, wrap with `>` and `< 0`
// The deposit uses FP64 atomics (the reference's GPU kernel races,
// src/pic.cu:124-127); the density is zeroed every step and forceOld starts at
// zero for every particle (the reference GPU path copies it with a grid-sized
// launch, src/pic.cu:574-575).  This file is compiled with --fmad=false so no
// multiply-add is contracted, as in the reference's x86 build.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include "pic_div_dev.cuh"
#include "pic_internal.cuh"

namespace pic {

struct CompatDev {
    int nx, ny, Y, nyh;      // padded rows of Y = ny + 2
    int lgx, lgy;            // powers of two: their logarithms (own transforms)
    double xDim, yDim;
    double dx, dy, area, q, qm, dt, hdt;  // hdt = dt / 2
    double rdx, rdy, rarea;  // 1/dx, 1/dy, 1/area, rounded to nearest
    double r2dx, r2dy;       // 1/(2 dx), 1/(2 dy)
    double norm;             // 1/(nx ny)
    long long np;
    double *px, *py, *vx, *vy;
    double *kox, *koy;       // dt/2 times the last force (the lagged half kick)
    double *w;               // four CIC weights per particle, planes of np, or null (KEPT)
    int2 *cell;
    double *rho;             // padded
    double2 *e;              // padded: Ex, Ey (ghosts stay zero)
    double *fin;             // nx x ny: the real transform's input and output
    cufftDoubleComplex *fout;  // half spectrum: [nx][nyh] for cuFFT, [nyh][nx] for the own transforms
    const double2 *twx, *twy;  // exp(-2 pi i k / n), n entries each
    double2 *kmode;          // -k^2 and its reciprocal (0, 0 for the zero mode), laid out as fout
};

// (int)(x / d) and its value as a double; positions in range take the
// integer from the low word of q + 2^52 rounded toward zero
__device__ __forceinline__ int cell_of(double x, double d, double rd, double &value)
{
    double q = div_known(x, d, rd);
    if ((unsigned)__double2hiint(q) < 0x41D00000u) {  // 0 <= q < 2^30
        const double t = __dadd_rz(q, 4503599627370496.0);
        value = __dsub_rn(t, 4503599627370496.0);
        return __double2loint(t);
    }
    const int c = (int)__ddiv_rn(x, d);
    value = (double)c;
    return c;
}

// X after a periodic step: X > dim ? X - dim : X < 0 ? X + dim : X, the
// comparisons on the bit patterns (integer pipe)
__device__ __forceinline__ double wrap_ref(double x, double dim)
{
    const long long b = __double_as_longlong(x);
    if (b > __double_as_longlong(dim)) return __dsub_rn(x, dim);
    if (b < 0 && b != (long long)0x8000000000000000ull) return __dadd_rn(x, dim);
    return x;
}

// CIC weights of a position in the cell whose indices are cx, cy
__device__ __forceinline__ void compat_weights(const CompatDev &D, double X, double Yp, double cx, double cy,
                                               double (&a)[4])
{
    const double bx = __dmul_rn(cx, D.dx), by = __dmul_rn(cy, D.dy);
    const double lx = __dsub_rn(X, bx), ly = __dsub_rn(Yp, by);
    const double hx = __dsub_rn(__dadd_rn(bx, D.dx), X), hy = __dsub_rn(__dadd_rn(by, D.dy), Yp);
    a[0] = div_known(__dmul_rn(lx, ly), D.area, D.rarea);
    a[1] = div_known(__dmul_rn(hx, ly), D.area, D.rarea);
    a[2] = div_known(__dmul_rn(lx, hy), D.area, D.rarea);
    a[3] = div_known(__dmul_rn(hx, hy), D.area, D.rarea);
}

// Cell and weights of a position, kept for the gather of the next push, and
// the particle's charge.  Cells run 0..nx (a particle exactly at x = xDim has
// cell nx); any other would index outside the padded grid: it is kept as it is
// and the particle skipped.
template <bool KEPT>
__device__ __forceinline__ void compat_place(const CompatDev &D, long long k, double X, double Yp)
{
    double cx, cy, a[4];
    const int ix = cell_of(X, D.dx, D.rdx, cx), iy = cell_of(Yp, D.dy, D.rdy, cy);
    D.cell[k] = make_int2(ix, iy);
    if ((unsigned)ix > (unsigned)D.nx || (unsigned)iy > (unsigned)D.ny) return;
    compat_weights(D, X, Yp, cx, cy, a);
    if (KEPT)
#pragma unroll
        for (int i = 0; i < 4; ++i) D.w[k + i * D.np] = a[i];
    const int ix1 = ix + 1 >= D.nx ? ix + 1 - D.nx : ix + 1, iy1 = iy + 1 >= D.ny ? iy + 1 - D.ny : iy + 1;
    double *r0 = D.rho + (size_t)(1 + ix) * D.Y, *r1 = D.rho + (size_t)(1 + ix1) * D.Y;
    atomicAdd(r0 + 1 + iy, __dmul_rn(a[0], D.q));
    atomicAdd(r1 + 1 + iy, __dmul_rn(a[1], D.q));
    atomicAdd(r0 + 1 + iy1, __dmul_rn(a[2], D.q));
    atomicAdd(r1 + 1 + iy1, __dmul_rn(a[3], D.q));
}

// Gather, lagged kick-drift-kick and the deposit of the new position for the
// next step, in one pass: the weights computed for the deposit are those of
// the next gather (32 bytes kept per particle instead of 24 FP64 operations).
// 128^2, 1.6 M particles: 220 us against 377 us for a push and 194 us for a
// deposit that each computed cells and weights with general divisions; 64
// FP64 operations per particle, 168 us at the pipe's rate.
// !KEPT: the weights are computed again for the gather (the same operations on
// the same position), where memory for them is short: 56 bytes per particle
// instead of 88.
template <bool DEPOSIT, bool KEPT>
__global__ void compat_push_kernel(CompatDev D)
{
    pdl_wait();
    pdl_trigger();
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= D.np) return;
    const int2 c = D.cell[k];
    if ((unsigned)c.x > (unsigned)D.nx || (unsigned)c.y > (unsigned)D.ny) return;
    const int ix1 = c.x + 1 >= D.nx ? c.x + 1 - D.nx : c.x + 1, iy1 = c.y + 1 >= D.ny ? c.y + 1 - D.ny : c.y + 1;
    const double2 *r0 = D.e + (size_t)c.x * D.Y, *r1 = D.e + (size_t)ix1 * D.Y;
    const double2 e1 = r0[c.y], e2 = r1[c.y], e3 = r0[iy1], e4 = r1[iy1];
    double a[4];
    if (KEPT)
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = D.w[k + i * D.np];
    else
        compat_weights(D, D.px[k], D.py[k], (double)c.x, (double)c.y, a);
    double fx = __dmul_rn(a[0], e1.x);
    fx = __dadd_rn(fx, __dmul_rn(a[1], e2.x));
    fx = __dadd_rn(fx, __dmul_rn(a[2], e3.x));
    fx = __dadd_rn(fx, __dmul_rn(a[3], e4.x));
    fx = __dmul_rn(fx, D.qm);
    double fy = __dmul_rn(a[0], e1.y);
    fy = __dadd_rn(fy, __dmul_rn(a[1], e2.y));
    fy = __dadd_rn(fy, __dmul_rn(a[2], e3.y));
    fy = __dadd_rn(fy, __dmul_rn(a[3], e4.y));
    fy = __dmul_rn(fy, D.qm);
    const double vxh = __dadd_rn(D.vx[k], D.kox[k]);
    const double vyh = __dadd_rn(D.vy[k], D.koy[k]);
    const double kox = __dmul_rn(D.hdt, fx), koy = __dmul_rn(D.hdt, fy);
    const double X = wrap_ref(__dadd_rn(D.px[k], __dmul_rn(vxh, D.dt)), D.xDim);
    const double Yp = wrap_ref(__dadd_rn(D.py[k], __dmul_rn(vyh, D.dt)), D.yDim);
    D.vx[k] = __dadd_rn(vxh, kox);
    D.vy[k] = __dadd_rn(vyh, koy);
    D.kox[k] = kox;
    D.koy[k] = koy;
    D.px[k] = X;
    D.py[k] = Yp;
    if (DEPOSIT) compat_place<KEPT>(D, k, X, Yp);
}

// Particle::Particle (particle.cc:21-29): cell from position, forces zero;
// and the first step's deposit.
template <bool KEPT>
__global__ void compat_setup_kernel(CompatDev D)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= D.np) return;
    D.kox[k] = 0.0;
    D.koy[k] = 0.0;
    compat_place<KEPT>(D, k, D.px[k], D.py[k]);
}

// Periodic ghost copy of a padded grid, two loops as the reference runs them
// (grid.cc:66-75 for rho with first = 0, fourier.cc:108-115 for phi with
// first = 1).  One block; the loops have no intra-loop dependencies.  Only
// the grids handed back need it: the solve reads the interior, the field is
// formed with periodic neighbours.
__global__ void compat_ghost_kernel(double *g, int nx, int ny, int first)
{
    const int Y = ny + 2, nxe = nx + 2, nye = ny + 2;
    const int last = first ? nye - 1 : nye;
    for (int i = first + threadIdx.x; i < last; i += blockDim.x) {
        g[i] = g[nx * Y + i];
        g[(nxe - 1) * Y + i] = g[Y + i];
    }
    __syncthreads();
    for (int i = 1 + threadIdx.x; i < nxe - 1; i += blockDim.x) {
        g[i * Y] = g[i * Y + ny];
        g[i * Y + (nye - 1)] = g[i * Y + 1];
    }
}

// -k^2 of every mode with the reference's wavenumbers, and its reciprocal
__global__ void compat_modes_kernel(CompatDev D)
{
    const double pi = 3.14159265358979323846;
    const bool own = D.lgx >= 0 && D.lgy >= 0;
    const int n = D.nx * D.nyh;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = own ? t % D.nx : t / D.nyh, j = own ? t / D.nx : t - i * D.nyh;
        const int II = (2 * i < D.nx) ? i : i - D.nx;
        const int JJ = (2 * j < D.nyh) ? j : j - D.ny;
        const double k1 = 2 * pi * II, k2 = 2 * pi * JJ;
        const double fact = __dadd_rn(__dmul_rn(k1, k1), __dmul_rn(k2, k2));
        D.kmode[t] = fabs(fact) < 1e-14 ? make_double2(0.0, 0.0) : make_double2(-fact, __ddiv_rn(1.0, -fact));
    }
}

// phi^ = -rho^ / k^2 of mode t (the zero mode removed)
__device__ __forceinline__ double2 compat_mode(const CompatDev &D, double2 o, int t)
{
    const double2 k = D.kmode[t];
    if (k.y == 0.0) return make_double2(0.0, 0.0);
    return make_double2(div_known(o.x, k.x, k.y), div_known(o.y, k.x, k.y));
}

// ---- sides that are no powers of two: cuFFT around these
__global__ void compat_pack_kernel(CompatDev D)
{
    pdl_wait();
    pdl_trigger();
    const int n = D.nx * D.ny;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = t / D.ny, j = t - i * D.ny;
        D.fin[t] = D.rho[(i + 1) * D.Y + (j + 1)];
    }
}

__global__ void compat_kspace_kernel(CompatDev D)
{
    pdl_wait();
    pdl_trigger();
    const int n = D.nx * D.nyh;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
        D.fout[t] = compat_mode(D, D.fout[t], t);
}

// ---- power-of-two sides: FP64 Stockham transforms in shared memory.  The
// FP64 pipe takes 64 cycles per warp instruction and SM partition, so a
// transform's time on a grid that does not fill the GPU is its instructions
// per warp: sides up to 128 give every component of every element its own thread and
// run radix 2 (three FP64 instructions per pass), larger ones run radix 4 on
// n/4 threads (half the operations).  128^2: 7.3 + 11.2 + 7.3 us (launched
// alone) for rows, columns and rows against 9.7 + 2 x 20.4 + 10.2 us in cuFFT
// and 4.8 us for the k-space operator; with the pack, unpack and ghost kernels
// gone, a step of 32^2 and 1600 particles went from 95 to 18 us.  tw[k] = exp(-2 pi i k / n), in shared
// memory.
constexpr int COMPAT_SPLIT_MAX = 7;  // log2 of the largest side with a thread per component
__host__ __device__ constexpr int compat_threads(int lg)
{
    return lg <= COMPAT_SPLIT_MAX ? 2 << lg : 1 << (lg - 2);
}

__device__ __forceinline__ double2 dcmul(double2 a, double2 w)
{
    return make_double2(__fma_rn(a.x, w.x, -__dmul_rn(a.y, w.y)),
                        __fma_rn(a.x, w.y, __dmul_rn(a.y, w.x)));
}

template <bool INV>
__device__ __forceinline__ double2 twiddle(const double2 *tw, int k)
{
    double2 w = tw[k];
    if (INV) w.y = -w.y;
    return w;
}

// The transform of x (n elements) by threads t of compat_threads(lg), with y
// as its second buffer; the result is left in x (the two pointers may have
// changed places).  Every thread of the block must call it; the input is
// complete after its first barrier.
template <bool INV>
__device__ void compat_fft(double2 *&x, double2 *&y, int lg, int t, const double2 *tw)
{
    const int n = 1 << lg;
    __syncthreads();
    if (lg <= COMPAT_SPLIT_MAX) {
        const int o = t >> 1, im = t & 1, h = n >> 1;
        for (int ln = 0; ln < lg; ++ln) {
            const int m = o & ((1 << ln) - 1), j = ((o >> (ln + 1)) << ln) + m;
            const double2 b = x[j + h], w = twiddle<INV>(tw, m << (lg - ln - 1));
            const double a = reinterpret_cast<const double *>(x + j)[im];
            const double p = im ? __fma_rn(b.x, w.y, __dmul_rn(b.y, w.x))
                                : __fma_rn(b.x, w.x, -__dmul_rn(b.y, w.y));
            reinterpret_cast<double *>(y + o)[im] = (o >> ln) & 1 ? __dsub_rn(a, p) : __dadd_rn(a, p);
            __syncthreads();
            double2 *const z = x;
            x = y;
            y = z;
        }
        return;
    }
    const int q = n >> 2;
    int ln = 0;  // log2 of the sub-transform length
    for (; ln + 2 <= lg; ln += 2) {
        const int m = t & ((1 << ln) - 1);
        double2 a = x[t], b = x[t + q], c = x[t + 2 * q], d = x[t + 3 * q];
        if (ln > 0) {
            const int st = m << (lg - ln - 2);
            b = dcmul(b, twiddle<INV>(tw, st));
            c = dcmul(c, twiddle<INV>(tw, 2 * st));
            d = dcmul(d, twiddle<INV>(tw, 3 * st));
        }
        const double2 s0 = make_double2(a.x + c.x, a.y + c.y), s1 = make_double2(a.x - c.x, a.y - c.y);
        const double2 s2 = make_double2(b.x + d.x, b.y + d.y);
        double2 s3 = make_double2(b.y - d.y, d.x - b.x);  // -i (b - d)
        if (INV) s3 = make_double2(-s3.x, -s3.y);
        const int o = ((t >> ln) << (ln + 2)) + m, ns = 1 << ln;
        __syncthreads();
        x[o] = make_double2(s0.x + s2.x, s0.y + s2.y);
        x[o + ns] = make_double2(s1.x + s3.x, s1.y + s3.y);
        x[o + 2 * ns] = make_double2(s0.x - s2.x, s0.y - s2.y);
        x[o + 3 * ns] = make_double2(s1.x - s3.x, s1.y - s3.y);
        __syncthreads();
    }
    if (ln < lg) {  // one bit left: butterflies t and t + n/4 of length n
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = t + h * q;
            const double2 a = x[j], b = dcmul(x[j + 2 * q], twiddle<INV>(tw, j));
            x[j] = make_double2(a.x + b.x, a.y + b.y);
            x[j + 2 * q] = make_double2(a.x - b.x, a.y - b.y);
        }
        __syncthreads();
    }
}

// shared memory of a block of `per` transforms of length n: the twiddles,
// then each transform's two buffers
__host__ __device__ constexpr size_t compat_smem(int n, int per)
{
    return sizeof(double2) * (size_t)n * (1 + 2 * per);
}

// twiddles into shared memory (before the wait: nothing in the chain writes them)
__device__ __forceinline__ void load_twiddles(double2 *s, const double2 *__restrict__ tw, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = __ldg(tw + i);
}

// Rows along the second index: two real rows per complex transform, split
// into their half spectra, written with the first index contiguous.
__global__ void __launch_bounds__(256) compat_rows_fwd_kernel(CompatDev D, int per)
{
    extern __shared__ double2 dsm[];
    const int n = D.ny, tp = compat_threads(D.lgy), f = threadIdx.x / tp, t = threadIdx.x - f * tp;
    const int i0 = 2 * (blockIdx.x * per + f);
    const bool on = f < per && i0 < D.nx;
    double2 *x = dsm + (1 + 2 * f) * n, *y = x + n;
    load_twiddles(dsm, D.twy, n);
    pdl_wait();
    pdl_trigger();
    const double *r0 = D.rho + (size_t)(i0 + 1) * D.Y + 1;
    if (on)
        for (int j = t; j < n; j += tp) x[j] = make_double2(r0[j], r0[D.Y + j]);
    compat_fft<false>(x, y, D.lgy, t, dsm);
    if (!on) return;
    for (int j = t; j < D.nyh; j += tp) {
        const double2 z = x[j], m = x[(n - j) & (n - 1)];
        double2 *o = (double2 *)D.fout + (size_t)j * D.nx + i0;
        o[0] = make_double2(0.5 * (z.x + m.x), 0.5 * (z.y - m.y));
        o[1] = make_double2(0.5 * (z.y + m.y), 0.5 * (m.x - z.x));
    }
}

// Columns along the first index: forward, the k-space operator, inverse, in place.
__global__ void __launch_bounds__(256) compat_cols_kernel(CompatDev D, int per)
{
    extern __shared__ double2 dsm[];
    const int n = D.nx, tp = compat_threads(D.lgx), f = threadIdx.x / tp, t = threadIdx.x - f * tp;
    const int j = blockIdx.x * per + f;
    const bool on = f < per && j < D.nyh;
    double2 *x = dsm + (1 + 2 * f) * n, *y = x + n;
    load_twiddles(dsm, D.twx, n);
    pdl_wait();
    pdl_trigger();
    double2 *col = (double2 *)D.fout + (size_t)j * n;
    if (on)
        for (int i = t; i < n; i += tp) x[i] = col[i];
    compat_fft<false>(x, y, D.lgx, t, dsm);
    if (on)
        for (int i = t; i < n; i += tp) x[i] = compat_mode(D, x[i], j * n + i);
    compat_fft<true>(x, y, D.lgx, t, dsm);
    if (on)
        for (int i = t; i < n; i += tp) col[i] = x[i];
}

// Rows back: two real rows per complex transform from their half spectra
// (the imaginary parts of the first and last mode dropped, as a complex-to-
// real transform does).
__global__ void __launch_bounds__(256) compat_rows_inv_kernel(CompatDev D, int per)
{
    extern __shared__ double2 dsm[];
    const int n = D.ny, tp = compat_threads(D.lgy), f = threadIdx.x / tp, t = threadIdx.x - f * tp;
    const int i0 = 2 * (blockIdx.x * per + f);
    const bool on = f < per && i0 < D.nx;
    double2 *x = dsm + (1 + 2 * f) * n, *y = x + n;
    load_twiddles(dsm, D.twy, n);
    pdl_wait();
    pdl_trigger();
    if (on)
        for (int j = t; j < D.nyh; j += tp) {
            const double2 *s = (const double2 *)D.fout + (size_t)j * D.nx + i0;
            double2 a = s[0], b = s[1];
            if (j == 0 || 2 * j == n) a.y = b.y = 0.0;
            x[j] = make_double2(a.x - b.y, a.y + b.x);
            if (j > 0 && 2 * j < n) x[n - j] = make_double2(a.x + b.y, b.x - a.y);
        }
    compat_fft<true>(x, y, D.lgy, t, dsm);
    if (!on) return;
    double *o = D.fin + (size_t)i0 * n;
    for (int j = t; j < n; j += tp) {
        o[j] = x[j].x;
        o[n + j] = x[j].y;
    }
}

// The field from the potential (periodic neighbours in place of its ghosts);
// with `clear` the density is zeroed for the next deposit.
__global__ void compat_efield_kernel(CompatDev D, int clear)
{
    pdl_wait();
    pdl_trigger();
    const int nx = D.nx, ny = D.ny, n = nx * ny, stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    auto phi = [&](int i, int j) { return __dmul_rn(__dmul_rn(D.fin[i * ny + j], D.norm), D.norm); };
    for (int t = t0; t < n; t += stride) {
        const int i = t / ny, j = t - i * ny;
        const int im = i ? i - 1 : nx - 1, ip = i + 1 < nx ? i + 1 : 0;
        const int jm = j ? j - 1 : ny - 1, jp = j + 1 < ny ? j + 1 : 0;
        D.e[(i + 1) * D.Y + (j + 1)] =
            make_double2(div_known(__dsub_rn(phi(i, jm), phi(i, jp)), 2 * D.dx, D.r2dx),
                         div_known(__dsub_rn(phi(im, j), phi(ip, j)), 2 * D.dy, D.r2dy));
    }
    if (clear)
        for (int t = t0; t < (nx + 2) * D.Y; t += stride) D.rho[t] = 0.0;
}

// The padded grids of the last step: phi, Ex, Ey.
__global__ void compat_unpack_kernel(CompatDev D, double *phi, double *ex, double *ey)
{
    const int n = (D.nx + 2) * D.Y;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = t / D.Y - 1, j = t - (i + 1) * D.Y - 1;
        const bool in = i >= 0 && i < D.nx && j >= 0 && j < D.ny;
        phi[t] = in ? __dmul_rn(__dmul_rn(D.fin[i * D.ny + j], D.norm), D.norm) : 0.0;
        ex[t] = D.e[t].x;
        ey[t] = D.e[t].y;
    }
}

static long long count_steps(double dt, double tmax)
{
    long long n = 0;
    double t = 0.0;
    while (t < tmax) {
        t += dt;
        ++n;
    }
    return n;
}

static pic_status compat_validate(const pic_ref_params *p)
{
    // main.cc:82 argument checks, plus the limits of this implementation
    if (!p || p->npx < 1 || p->npy < 1 || p->xDim <= 0 || p->yDim <= 0 || p->nx < 2 ||
        p->ny < 2 || !(p->dt > 0.0) || p->tmax < 0.0 || !(p->mass != 0.0) ||
        (long long)p->nx * p->ny > (1ll << 26)) {
        set_error("pic_compat_run: invalid reference parameters");
        return PIC_ERR_INVALID_ARG;
    }
    return PIC_OK;
}

namespace {
struct CompatRun {
    CompatDev D{};
    cufftHandle fwd = 0, inv = 0;
    cudaStream_t st = nullptr;
    std::vector<void *> allocs;
    ~CompatRun()
    {
        if (fwd) cufftDestroy(fwd);
        if (inv) cufftDestroy(inv);
        for (void *a : allocs) cudaFree(a);
        if (st) cudaStreamDestroy(st);
    }
    template <class T> pic_status alloc(T **p, size_t n)
    {
        void *q = nullptr;
        PIC_CUDA(cudaMalloc(&q, n * sizeof(T)));
        allocs.push_back(q);
        *p = (T *)q;
        return PIC_OK;
    }
};

// log2 of a side the own transforms take (8..1024), or -1
int compat_log2(int n)
{
    for (int l = 3; l <= 10; ++l)
        if (n == 1 << l) return l;
    return -1;
}

// transforms of length 2^lg per block: about one block per SM, at most 256 threads
int compat_per_block(int lg, int items)
{
    int k = 1;
    while (2 * k <= std::min(256 / compat_threads(lg), items / device_sms())) k *= 2;
    return k;
}

// rho (padded) -> fin (the potential before its normalisation)
pic_status compat_solve(CompatRun &R)
{
    CompatDev &D = R.D;
    if (D.lgx < 0 || D.lgy < 0) {
        const int gg = grid_for((long long)D.nx * D.ny, 256);
        void *args[] = {&D};
        PIC_TRY(launch_dependent((const void *)compat_pack_kernel, gg, 256, 0, R.st, args));
        PIC_CUFFT(cufftExecD2Z(R.fwd, D.fin, D.fout));
        PIC_TRY(launch_dependent((const void *)compat_kspace_kernel, gg, 256, 0, R.st, args));
        PIC_CUFFT(cufftExecZ2D(R.inv, D.fout, D.fin));
        return PIC_OK;
    }
    int pr = compat_per_block(D.lgy, D.nx / 2), pc = compat_per_block(D.lgx, D.nyh);
    const unsigned br = (D.nx / 2 + pr - 1) / pr, bc = (D.nyh + pc - 1) / pc;
    const int tr = pr * compat_threads(D.lgy), tc = pc * compat_threads(D.lgx);
    const size_t mr = compat_smem(D.ny, pr), mc = compat_smem(D.nx, pc);
    void *ar[] = {&D, &pr}, *ac[] = {&D, &pc};
    PIC_TRY(launch_dependent((const void *)compat_rows_fwd_kernel, br, tr, mr, R.st, ar));
    PIC_TRY(launch_dependent((const void *)compat_cols_kernel, bc, tc, mc, R.st, ac));
    return launch_dependent((const void *)compat_rows_inv_kernel, br, tr, mr, R.st, ar);
}
}  // namespace

static pic_status compat_core(const pic_ref_params *p, const double *x0, const double *y0,
                              const double *vx0, const double *vy0, long long nsteps, double *x,
                              double *y, double *vx, double *vy, double *rho, double *phi,
                              double *ex, double *ey)
{
    PIC_TRY(compat_validate(p));
    if (!x0 || !y0 || !vx0 || !vy0 || nsteps < 0) {
        set_error("pic_compat_run: null input array or negative step count");
        return PIC_ERR_INVALID_ARG;
    }
    CompatRun R;
    CompatDev &D = R.D;
    D.nx = p->nx;
    D.ny = p->ny;
    D.Y = p->ny + 2;
    D.nyh = p->ny / 2 + 1;
    D.lgx = compat_log2(p->nx);
    D.lgy = compat_log2(p->ny);
    D.xDim = p->xDim;
    D.yDim = p->yDim;
    D.dx = (double)p->xDim / p->nx;  // main.cc:75-77
    D.dy = (double)p->yDim / p->ny;
    D.area = D.dx * D.dy;
    D.rdx = 1.0 / D.dx;
    D.rdy = 1.0 / D.dy;
    D.rarea = 1.0 / D.area;
    D.r2dx = 1.0 / (2 * D.dx);
    D.r2dy = 1.0 / (2 * D.dy);
    D.norm = 1.0 / (p->nx * p->ny);
    D.q = p->charge;
    D.qm = p->charge / p->mass;
    D.dt = p->dt;
    D.hdt = 0.5 * p->dt;
    D.np = (long long)p->npx * p->npy;
    const size_t np = (size_t)D.np, ng = (size_t)(p->nx + 2) * D.Y, n = (size_t)p->nx * p->ny;
    PIC_CUDA(cudaStreamCreateWithFlags(&R.st, cudaStreamNonBlocking));
    // on 16-byte boundaries: field (padded), spectrum, twiddles and the real
    // transforms' grid (cuFFT wants it so); then cells and doubles
    const size_t nk = (size_t)p->nx * D.nyh, n16 = ng + 2 * nk + p->nx + p->ny + (n + 1) / 2;
    double2 *pool16 = nullptr;
    double *pool = nullptr;
    PIC_TRY(R.alloc(&pool16, n16));
    // the weights (4 np) only where they fit the device and the caller's budget
    const size_t lean = 7 * np + 4 * ng;
    bool kept = stage_budget((lean + 4 * np) * sizeof(double));
    if (kept && R.alloc(&pool, lean + 4 * np) != PIC_OK) {
        cudaGetLastError();
        kept = false;
    }
    if (!kept) PIC_TRY(R.alloc(&pool, lean));
    D.e = pool16;
    D.fout = (cufftDoubleComplex *)(D.e + ng);
    D.kmode = (double2 *)D.fout + nk;
    double2 *tw = D.kmode + nk;
    D.twx = tw;
    D.twy = tw + p->nx;
    D.cell = (int2 *)pool;
    D.px = pool + np;
    D.py = D.px + np;
    D.vx = D.py + np;
    D.vy = D.vx + np;
    D.kox = D.vy + np;
    D.koy = D.kox + np;
    D.w = kept ? D.koy + np : nullptr;
    D.rho = D.koy + (kept ? 5 : 1) * np;
    double *dphi = D.rho + ng, *dex = dphi + ng, *dey = dex + ng;
    D.fin = (double *)(tw + p->nx + p->ny);
    PIC_CUDA(cudaMemsetAsync(D.e, 0, sizeof(double2) * ng, R.st));
    PIC_CUDA(cudaMemsetAsync(D.rho, 0, sizeof(double) * ng, R.st));
    PIC_CUDA(cudaMemsetAsync(D.fin, 0, sizeof(double) * n, R.st));
    PIC_CUDA(cudaMemcpyAsync(D.px, x0, sizeof(double) * np, cudaMemcpyHostToDevice, R.st));
    PIC_CUDA(cudaMemcpyAsync(D.py, y0, sizeof(double) * np, cudaMemcpyHostToDevice, R.st));
    PIC_CUDA(cudaMemcpyAsync(D.vx, vx0, sizeof(double) * np, cudaMemcpyHostToDevice, R.st));
    PIC_CUDA(cudaMemcpyAsync(D.vy, vy0, sizeof(double) * np, cudaMemcpyHostToDevice, R.st));
    std::vector<double2> htw;
    if (D.lgx >= 0 && D.lgy >= 0) {
        for (int s : {p->nx, p->ny})
            for (int k = 0; k < s; ++k) {
                const long double a = 2.0L * 3.14159265358979323846264338327950288L * k / s;
                htw.push_back(make_double2((double)std::cos(a), (double)-std::sin(a)));
            }
        PIC_CUDA(cudaMemcpyAsync(tw, htw.data(), sizeof(double2) * htw.size(), cudaMemcpyHostToDevice, R.st));
    } else {
        PIC_CUFFT(cufftPlan2d(&R.fwd, p->nx, p->ny, CUFFT_D2Z));
        PIC_CUFFT(cufftPlan2d(&R.inv, p->nx, p->ny, CUFFT_Z2D));
        PIC_CUFFT(cufftSetStream(R.fwd, R.st));
        PIC_CUFFT(cufftSetStream(R.inv, R.st));
    }
    // small runs on one-warp blocks: one FP64 partition each
    const int bt = D.np < 256ll * device_sms() ? 32 : 256;
    const unsigned gp = (unsigned)((D.np + bt - 1) / bt);
    const int gg = grid_for((long long)n, 256);
    if (nsteps > 0) {
        compat_modes_kernel<<<grid_for((long long)nk, 256), 256, 0, R.st>>>(D);
        if (kept)
            compat_setup_kernel<true><<<gp, bt, 0, R.st>>>(D);
        else
            compat_setup_kernel<false><<<gp, bt, 0, R.st>>>(D);
        PIC_CUDA(cudaGetLastError());
    }
    for (long long s = 0; s < nsteps; ++s) {
        PIC_TRY(compat_solve(R));
        int more = s + 1 < nsteps;
        void *ae[] = {&D, &more}, *ap[] = {&D};
        PIC_TRY(launch_dependent((const void *)compat_efield_kernel, gg, 256, 0, R.st, ae));
        const void *push = kept ? (more ? (const void *)compat_push_kernel<true, true>
                                        : (const void *)compat_push_kernel<false, true>)
                                : (more ? (const void *)compat_push_kernel<true, false>
                                        : (const void *)compat_push_kernel<false, false>);
        PIC_TRY(launch_dependent(push, gp, bt, 0, R.st, ap));
    }
    // the last step's grids
    compat_ghost_kernel<<<1, 1024, 0, R.st>>>(D.rho, D.nx, D.ny, 0);
    compat_unpack_kernel<<<grid_for((long long)ng, 256), 256, 0, R.st>>>(D, dphi, dex, dey);
    compat_ghost_kernel<<<1, 1024, 0, R.st>>>(dphi, D.nx, D.ny, 1);
    PIC_CUDA(cudaGetLastError());
    if (x) PIC_CUDA(cudaMemcpyAsync(x, D.px, sizeof(double) * np, cudaMemcpyDeviceToHost, R.st));
    if (y) PIC_CUDA(cudaMemcpyAsync(y, D.py, sizeof(double) * np, cudaMemcpyDeviceToHost, R.st));
    if (vx) PIC_CUDA(cudaMemcpyAsync(vx, D.vx, sizeof(double) * np, cudaMemcpyDeviceToHost, R.st));
    if (vy) PIC_CUDA(cudaMemcpyAsync(vy, D.vy, sizeof(double) * np, cudaMemcpyDeviceToHost, R.st));
    if (rho) PIC_CUDA(cudaMemcpyAsync(rho, D.rho, sizeof(double) * ng, cudaMemcpyDeviceToHost, R.st));
    if (phi) PIC_CUDA(cudaMemcpyAsync(phi, dphi, sizeof(double) * ng, cudaMemcpyDeviceToHost, R.st));
    if (ex) PIC_CUDA(cudaMemcpyAsync(ex, dex, sizeof(double) * ng, cudaMemcpyDeviceToHost, R.st));
    if (ey) PIC_CUDA(cudaMemcpyAsync(ey, dey, sizeof(double) * ng, cudaMemcpyDeviceToHost, R.st));
    PIC_CUDA(cudaStreamSynchronize(R.st));
    return PIC_OK;
}

}  // namespace pic

extern "C" pic_status pic_compat_run_steps(const pic_ref_params *p, const double *x0,
                                           const double *y0, const double *vx0,
                                           const double *vy0, long long nsteps, double *x,
                                           double *y, double *vx, double *vy, double *rho,
                                           double *phi, double *ex, double *ey)
{
    return pic::compat_core(p, x0, y0, vx0, vy0, nsteps, x, y, vx, vy, rho, phi, ex, ey);
}

extern "C" pic_status pic_compat_run(const pic_ref_params *p, const double *posX,
                                     const double *posY, const double *velX, const double *velY,
                                     double *xOut, double *yOut, double *seconds)
{
    PIC_TRY(pic::compat_validate(p));
    const auto t0 = std::chrono::steady_clock::now();
    const long long nsteps = pic::count_steps(p->dt, p->tmax);
    pic_status s = pic::compat_core(p, posX, posY, velX, velY, nsteps, xOut, yOut, nullptr,
                                    nullptr, nullptr, nullptr, nullptr, nullptr);
    const auto t1 = std::chrono::steady_clock::now();
    if (seconds) *seconds = std::chrono::duration<double>(t1 - t0).count();
    return s;
}
