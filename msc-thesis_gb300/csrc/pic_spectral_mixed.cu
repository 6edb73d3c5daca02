// pic_spectral_mixed.cu -- the spectral field solve of grids whose sides are
// products of 2, 3, 5 and 7 (not both powers of two): three kernels, rows,
// columns and rows, as in pic_spectral.cu.
//
// These grids went through cuFFT: conversion, two transform kernels, the
// k-space kernel and four more transform kernels, each a few us of launch and
// latency.  Here the conversion, the k-space operator, the clearing of the
// density and the diagnostics fold ride on the three kernels; the spectra
// between them lie in memory ([mode][row]).  A transform is a list of Stockham
// passes of radix 2 to 10 between two shared buffers, the host choosing the
// fewest passes; a block holds one transform (or few), so that the chain of a
// kernel is about three passes of one butterfly a thread.  The inverse
// transforms run as forward ones on values whose real and imaginary parts are
// swapped, so that there is one copy of the passes.  Bound by launches and those
// chains up to about 256 a side.  One step with 23 particles per cell, cuFFT ->
// here: 60x60 22.3 -> 15.7 us, 96x96 25.1 -> 17.3, 250x180 35.4 -> 26.0, 500x500
// 102 -> 78, 1000x1000 246 -> 242.  All of it in one cluster of eight blocks, as
// the small powers of two: 15.2, 18.5 and 36 us for the first three.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "pic_spectral_dev.cuh"

namespace pic {
namespace {

constexpr int MAX_PASSES = 8;  // 256 = 2^8
constexpr int MAX_SIDE = 1024;
constexpr size_t MAX_SMEM = 220 * 1024;

// w / d for w < 2^16, 1 < d <= 2^10, by the rounded-up reciprocal inv = ceil(2^32 / d):
// w (inv d - 2^32) < 2^16 2^10 < 2^32, so the error never reaches the next integer
__host__ inline unsigned reciprocal(int d) { return d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u; }
__device__ __forceinline__ int quotient(int w, unsigned inv) { return inv ? (int)__umulhi((unsigned)w, inv) : w; }

struct MixPass {
    int R, NS, M;              // radix, length of the sub-transforms, butterflies N / R
    int step;                  // N / (R NS): twiddle of output r, position m is W_N^(r m step)
    unsigned inv_m, inv_ns;
};
struct MixDim {
    int passes;
    MixPass p[MAX_PASSES];
};
struct MixArgs {
    SpecArgs A;
    MixDim dx, dy;
    int sx, sy;                // strides of the row and the column buffers
    int np, nc, nr;            // row pairs, columns, rows of a block (the last ones have fewer)
    unsigned inv_nx, inv_ny, inv_npair, inv_nr;
};

// X_k = sum_n x_n W_P^(n k), P = 3, 5 or 7: pairs x_n +- x_(P-n) share their
// cosine and sine sums
template <int P>
__device__ __forceinline__ void dft_odd(float2 *v)
{
    constexpr int H = P / 2;
    // cos, sin of 2 pi k / P, k = 1..H
    constexpr float c3[1] = {-0.5f}, s3[1] = {0.86602540378443864676f};
    constexpr float c5[2] = {0.30901699437494742410f, -0.80901699437494742410f};
    constexpr float s5[2] = {0.95105651629515357212f, 0.58778525229247312917f};
    constexpr float c7[3] = {0.62348980185873353053f, -0.22252093395631440429f, -0.90096886790241912624f};
    constexpr float s7[3] = {0.78183148246802980871f, 0.97492791218182360702f, 0.43388373911755812048f};
    float2 a[H], d[H], z = v[0];
#pragma unroll
    for (int n = 0; n < H; ++n) {
        a[n] = fft::cadd(v[1 + n], v[P - 1 - n]);
        d[n] = fft::csub(v[1 + n], v[P - 1 - n]);
        z = fft::cadd(z, a[n]);
    }
    float2 u[P];
    u[0] = z;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 m = v[0], s = make_float2(0.f, 0.f);
#pragma unroll
        for (int n = 1; n <= H; ++n) {
            const int e = (n * k) % P;            // angle 2 pi e / P
            const int f = (e <= H ? e : P - e) - 1;
            const float c = P == 3 ? c3[P == 3 ? f : 0] : P == 5 ? c5[P == 5 ? f : 0] : c7[P == 7 ? f : 0];
            const float w0 = P == 3 ? s3[P == 3 ? f : 0] : P == 5 ? s5[P == 5 ? f : 0] : s7[P == 7 ? f : 0];
            const float w = e <= H ? w0 : -w0;
            m.x = fmaf(c, a[n - 1].x, m.x);
            m.y = fmaf(c, a[n - 1].y, m.y);
            s.x = fmaf(w, d[n - 1].x, s.x);
            s.y = fmaf(w, d[n - 1].y, s.y);
        }
        u[k] = make_float2(m.x + s.y, m.y - s.x);      // m - i s
        u[P - k] = make_float2(m.x - s.y, m.y + s.x);  // m + i s
    }
#pragma unroll
    for (int k = 0; k < P; ++k) v[k] = u[k];
}

// forward DFT of v[0, R); 6 = 2 x 3 and 10 = 2 x 5 by coprime factors, without twiddles
template <int R>
__device__ __forceinline__ void dft_mixed(float2 *v)
{
    if constexpr (R == 3 || R == 5 || R == 7) {
        dft_odd<R>(v);
    } else if constexpr (R == 6 || R == 10) {
        constexpr int Q = R / 2;
        // input (Q n1 + 2 n2) mod R; output k with k mod 2 = k1, k mod Q = k2
        float2 e[Q], o[Q];
#pragma unroll
        for (int n = 0; n < Q; ++n) {
            const float2 x = v[(2 * n) % R], y = v[(Q + 2 * n) % R];
            e[n] = fft::cadd(x, y);
            o[n] = fft::csub(x, y);
        }
        dft_odd<Q>(e);
        dft_odd<Q>(o);
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = (k & 1) ? o[k % Q] : e[k % Q];
    } else {
        fft::dft<R, false>(v);
    }
}

// one pass over `count` transforms of stride S, from slot src to slot dst
template <int R, int T>
__device__ __forceinline__ void mix_pass(float2 *smem, int src, int dst, int count, int S,
                                         const MixPass &P, const float2 *tw)
{
    const int total = count * P.M;
    for (int w = threadIdx.x; w < total; w += T) {
        const int f = quotient(w, P.inv_m), j = w - f * P.M;
        const int q = quotient(j, P.inv_ns), m = P.NS > 1 ? j - q * P.NS : 0;
        const float2 *const in = smem + src + f * S + j;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = in[r * P.M];
        if (P.NS > 1) {
            const int ms = m * P.step;
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = fft::cmul(v[r], tw[r * ms]);
        }
        dft_mixed<R>(v);
        float2 *const out = smem + dst + f * S + q * P.NS * R + m;
#pragma unroll
        for (int r = 0; r < R; ++r) out[r * P.NS] = v[r];
    }
}

__shared__ MixDim s_dim[2];  // the plans along x and y

// forward transforms of `count` sequences at slot a;
// returns the slot that holds the results, a or b, behind a barrier
template <int T>
__device__ __noinline__ int run_passes(int dim, int a, int b, int count, int S, int tw)
{
    extern __shared__ __align__(16) float2 smem[];
    const MixDim &D = s_dim[dim];
    for (int i = 0; i < D.passes; ++i) {
        const MixPass P = D.p[i];
        __syncthreads();
        switch (P.R) {
        case 2: mix_pass<2, T>(smem, a, b, count, S, P, smem + tw); break;
        case 3: mix_pass<3, T>(smem, a, b, count, S, P, smem + tw); break;
        case 4: mix_pass<4, T>(smem, a, b, count, S, P, smem + tw); break;
        case 5: mix_pass<5, T>(smem, a, b, count, S, P, smem + tw); break;
        case 6: mix_pass<6, T>(smem, a, b, count, S, P, smem + tw); break;
        case 7: mix_pass<7, T>(smem, a, b, count, S, P, smem + tw); break;
        case 8: mix_pass<8, T>(smem, a, b, count, S, P, smem + tw); break;
        default: mix_pass<10, T>(smem, a, b, count, S, P, smem + tw); break;
        }
        const int t = a;
        a = b;
        b = t;
    }
    __syncthreads();
    return a;
}

__device__ __forceinline__ void load_plans(const MixArgs &G)
{
    if (threadIdx.x < MAX_PASSES) {
        s_dim[0].p[threadIdx.x] = G.dx.p[threadIdx.x];
        s_dim[1].p[threadIdx.x] = G.dy.p[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        s_dim[0].passes = G.dx.passes;
        s_dim[1].passes = G.dy.passes;
    }
}

template <int T>
__global__ void __launch_bounds__(T) mix_rows_fwd_kernel(const __grid_constant__ MixArgs G)
{
    extern __shared__ __align__(16) float2 smem[];
    const SpecArgs &A = G.A;
    const int nx = A.nx, ny = A.ny, nh = A.nh, b = G.np * G.sx, tw = 2 * b;
    for (int j = threadIdx.x; j < nx; j += T) smem[tw + j] = __ldg(A.twx + j);
    load_plans(G);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const int p0 = blockIdx.x * G.np, np = min(G.np, (ny + 1) / 2 - p0);
    unsigned long long qs = 0;
    for (int w = threadIdx.x; w < np * nx; w += T) {
        const int f = quotient(w, G.inv_nx);
        const size_t c = (size_t)(2 * p0 + f) * nx + w;  // row 2 (p0 + f)
        const bool two = 2 * (p0 + f) + 1 < ny;
        const unsigned long long a = __ldcg(A.rho_fix + c), d = two ? __ldcg(A.rho_fix + c + nx) : 0ull;
        qs += a + d;
        const float fa = fixed_to_float(a, A.mean_fix, A.scale);
        const float fd = two ? fixed_to_float(d, A.mean_fix, A.scale) : 0.f;
        A.rho[c] = fa;
        if (two) A.rho[c + nx] = fd;
        smem[f * G.sx + w - f * nx] = make_float2(fa, fd);
    }
    const int buf = run_passes<T>(0, 0, b, np, G.sx, tw);
    for (int w = threadIdx.x; w < nh * G.np; w += T) {
        // the pair fastest: a mode's rows are neighbours
        const int k = quotient(w, G.inv_npair), f = w - k * G.np;
        if (f >= np) continue;
        const float2 *const bb = smem + buf + f * G.sx;
        const float2 z = bb[k], m = bb[k ? nx - k : 0];
        float2 *const to = A.S + (size_t)k * ny + 2 * (p0 + f);
        to[0] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
        if (2 * (p0 + f) + 1 < ny) to[1] = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
    }
    qs = warp_sum(qs);
    if ((threadIdx.x & 31) == 0) atomicAdd(&A.dev->q[acc_slot()], qs);
}

template <int T>
__global__ void __launch_bounds__(T) mix_cols_kernel(const __grid_constant__ MixArgs G)
{
    extern __shared__ __align__(16) float2 smem[];
    const SpecArgs &A = G.A;
    const int nx = A.nx, ny = A.ny, b = 2 * G.nc * G.sy, tw = 2 * b;
    for (int j = threadIdx.x; j < ny; j += T) smem[tw + j] = __ldg(A.twx + nx + j);
    load_plans(G);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    // the density, converted by the forward rows, cleared for the next deposit
    for (int i = blockIdx.x * T + threadIdx.x; i < nx * ny; i += gridDim.x * T) A.rho_fix[i] = 0ull;
    const int c0 = blockIdx.x * G.nc, nc = min(G.nc, A.nh - c0);
    for (int w = threadIdx.x; w < nc * ny; w += T) {
        const int f = quotient(w, G.inv_ny);
        smem[f * G.sy + w - f * ny] = __ldcg(A.S + (size_t)c0 * ny + w);
    }
    int buf = run_passes<T>(1, 0, b, nc, G.sy, tw);
    float fe = 0.f;
    for (int w = threadIdx.x; w < nc * ny; w += T) {
        const int f = quotient(w, G.inv_ny), my = w - f * ny, mx = c0 + f;
        float2 *const at = smem + buf + f * G.sy + my;
        const float2 r = *at;
        const KMode K = kspace_mode(r, mx, my, nx, ny, A.kx1, A.ky1, A.inv_eps0_n, mx == 0 && my == 0);
        at[0] = make_float2(K.ph.y, K.ph.x);
        at[nc * G.sy] = make_float2(K.ey.y, K.ey.x);
        fe += K.fe;
        if (mx == A.tmx && my == A.tmy) {
            const double x = r.x, y = r.y;
            A.dev->mode_amp = sqrt(x * x + y * y) / ((double)nx * ny);
        }
    }
    buf = run_passes<T>(1, buf, b - buf, 2 * nc, G.sy, tw);
    for (int w = threadIdx.x; w < nc * ny; w += T) {
        const int f = quotient(w, G.inv_ny), y = w - f * ny, mx = c0 + f;
        const float2 p = smem[buf + f * G.sy + y], e = smem[buf + (f + nc) * G.sy + y];
        const float kxe = (2 * mx == nx) ? 0.f : A.kx1 * (float)mx;
        A.Tx[(size_t)c0 * ny + w] = make_float2(kxe * p.x, -kxe * p.y);
        A.Ty[(size_t)c0 * ny + w] = make_float2(e.y, e.x);
    }
    const double sum = warp_sum((double)fe);
    if ((threadIdx.x & 31) == 0) atomicAdd(&A.dev->fe[acc_slot()], sum);
}

template <int T>
__global__ void __launch_bounds__(T) mix_rows_inv_kernel(const __grid_constant__ MixArgs G)
{
    extern __shared__ __align__(16) float2 smem[];
    const SpecArgs &A = G.A;
    const int nx = A.nx, ny = A.ny, nh = A.nh, b = G.nr * G.sx, tw = 2 * b;
    for (int j = threadIdx.x; j < nx; j += T) smem[tw + j] = __ldg(A.twx + j);
    load_plans(G);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    if (A.adv && blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x < 32) advance_state(A.dev, A.hist, A.hist_cap, A.adv, A.fe_scale, 32);
        return;
    }
    const int y0 = blockIdx.x * G.nr, nr = min(G.nr, ny - y0);
    for (int w = threadIdx.x; w < nh * G.nr; w += T) {
        // the row fastest: a mode's rows are neighbours
        const int k = quotient(w, G.inv_nr), f = w - k * G.nr;
        if (f >= nr) continue;
        float2 x = __ldcg(A.Tx + (size_t)k * ny + y0 + f), y = __ldcg(A.Ty + (size_t)k * ny + y0 + f);
        if (k == 0 || 2 * k == nx) x.y = y.y = 0.f;
        float2 *const bb = smem + f * G.sx;
        bb[k] = make_float2(x.y + y.x, x.x - y.y);
        if (k > 0 && 2 * k != nx) bb[nx - k] = make_float2(y.x - x.y, x.x + y.y);
    }
    const int buf = run_passes<T>(0, 0, b, nr, G.sx, tw);
    for (int w = threadIdx.x; w < nr * nx; w += T) {
        const int f = quotient(w, G.inv_nx);
        const float2 v = smem[buf + f * G.sx + w - f * nx];
        A.ex[(size_t)y0 * nx + w] = v.y;
        A.ey[(size_t)y0 * nx + w] = v.x;
    }
}

// ---------------------------------------------------------------- host
// the fewest passes whose radices multiply to n, odd radices first (their
// stores of the first pass meet no bank conflicts); false: other factors
bool factor(int n, std::vector<int> &best)
{
    static const int radix[] = {10, 8, 7, 6, 5, 4, 3, 2};
    best.clear();
    std::vector<int> cur;
    int best_sum = 0;
    auto go = [&](auto &&self, int rest, int from) -> void {
        if (!best.empty() && cur.size() + (rest > 1) > best.size()) return;
        if (rest == 1) {
            int sum = 0;
            for (int r : cur) sum += r;
            if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && sum < best_sum)) {
                best = cur;
                best_sum = sum;
            }
            return;
        }
        if ((int)cur.size() == MAX_PASSES) return;
        for (int i = from; i < 8; ++i)
            if (rest % radix[i] == 0) {
                cur.push_back(radix[i]);
                self(self, rest / radix[i], i);
                cur.pop_back();
            }
    };
    go(go, n, 0);
    std::stable_sort(best.begin(), best.end(), [](int a, int b) { return (a & 1) > (b & 1); });
    return !best.empty();
}

bool plan_dim(int n, MixDim &D)
{
    std::vector<int> r;
    if (n < 2 || n > MAX_SIDE || !factor(n, r)) return false;
    D.passes = (int)r.size();
    int ns = 1;
    for (int i = 0; i < D.passes; ++i) {
        MixPass &P = D.p[i];
        P.R = r[i];
        P.NS = ns;
        P.M = n / P.R;
        P.step = n / (P.R * ns);
        P.inv_m = reciprocal(P.M);
        P.inv_ns = reciprocal(ns);
        ns *= P.R;
    }
    return true;
}

// false: sides that the kernels do not take
bool plan(int nx, int ny, MixArgs &G, size_t (&smem)[3])
{
    memset(&G, 0, sizeof G);
    if (nx < 16 || ny < 16 || !plan_dim(nx, G.dx) || !plan_dim(ny, G.dy)) return false;
    // at most four blocks per SM (two: 700x640 129 us a step, four: 122); on 152
    // SMs that is one row pair and one column a block for every side taken here,
    // and one row back or two
    const int blocks = 4 * device_sms();
    auto share = [&](int items) { return (items + blocks - 1) / blocks; };
    G.np = share((ny + 1) / 2);
    G.nc = share(nx / 2 + 1);
    G.nr = share(ny);
    G.sx = nx | 1;  // odd: lanes on different transforms use different banks
    G.sy = ny | 1;
    G.inv_nx = reciprocal(nx);
    G.inv_ny = reciprocal(ny);
    G.inv_npair = reciprocal(G.np);
    G.inv_nr = reciprocal(G.nr);
    smem[0] = sizeof(float2) * (2 * (size_t)G.np * G.sx + nx);
    smem[1] = sizeof(float2) * (4 * (size_t)G.nc * G.sy + ny);
    smem[2] = sizeof(float2) * (2 * (size_t)G.nr * G.sx + nx);
    return std::max({smem[0], smem[1], smem[2]}) <= MAX_SMEM;
}

}  // namespace

bool mixed_wanted(int nx, int ny)
{
    const char *solver = getenv("PIC_FIELD_SOLVER");
    if (solver && strcmp(solver, "cufft") == 0) return false;
    MixArgs G;
    size_t smem[3];
    return !spectral_size_ok(nx, ny) && plan(nx, ny, G, smem);
}

pic_status mixed_twiddles(int nx, int ny, float2 **tw)
{
    const double pi = 3.14159265358979323846;
    std::vector<float2> t;
    for (int n : {nx, ny})
        for (int j = 0; j < n; ++j) {
            const double a = 2.0 * pi * (double)j / (double)n;
            t.push_back(make_float2((float)std::cos(a), (float)-std::sin(a)));
        }
    PIC_CUDA(cudaMalloc(tw, t.size() * sizeof(float2)));
    PIC_CUDA(cudaMemcpy(*tw, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice));
    return PIC_OK;
}

pic_status launch_mixed(pic_handle *h, int adv)
{
    MixArgs G;
    size_t smem[3];
    if (!plan(h->g.nx, h->g.ny, G, smem)) {
        set_error("mixed-radix solve: grid sides");
        return PIC_ERR_INVALID_ARG;
    }
    spectral_args(h, adv, nullptr, G.A);
    void *args[] = {&G};
    // threads: a butterfly each for sides of about T, more for the longer
    // transforms (250x180 26.5 us a step with 128, 25.9 with 256; 48x200 18.4
    // and 21.0, 360x350 45.2 and 45.8, 700x640 142 and 129)
    const bool wide = (long long)h->g.nx * h->g.ny >= 32768;
    const int T = wide ? 256 : 128;
    const void *const kernel[3] = {
        wide ? (const void *)mix_rows_fwd_kernel<256> : (const void *)mix_rows_fwd_kernel<128>,
        wide ? (const void *)mix_cols_kernel<256> : (const void *)mix_cols_kernel<128>,
        wide ? (const void *)mix_rows_inv_kernel<256> : (const void *)mix_rows_inv_kernel<128>};
    const int items[3] = {(h->g.ny + 1) / 2, h->g.nh, h->g.ny}, per[3] = {G.np, G.nc, G.nr};
    for (int k = 0; k < 3; ++k) {
        const int blocks = (items[k] + per[k] - 1) / per[k] + (k == 2 && adv ? 1 : 0);
        PIC_TRY(allow_dynamic_smem(kernel[k], smem[k]));
        PIC_TRY(launch_dependent(kernel[k], dim3(blocks), dim3(T), smem[k], h->stream, args));
    }
    return PIC_OK;
}

}  // namespace pic
