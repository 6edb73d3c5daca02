// pic_spectral.cu -- the step's Poisson solve for power-of-two grids
// (16..4096 cells a side) in three hand-written kernels instead of the
// conversion kernel, two cuFFT transforms and the k-space kernel.  (Sides of
// 32 to 128 run the same operations in one kernel, pic_spectral_small.cu;
// other sides with factors 2, 3, 5 and 7 in pic_spectral_mixed.cu.)
//
//   rows_fwd  fixed-point density -> float rho (background removed, charge
//             summed), then the real FFT of each row along x: two rows per
//             complex transform (z = rho_a + i rho_b; A_k = (Z_k + conj
//             Z_-k) / 2, B_k = (Z_k - conj Z_-k) / 2i), modes 0..nx/2 of
//             every row written column-major, S[kx][y];
//   cols      per column kx: FFT along y, the k-space operator of the
//             conversion-free solve (phi^ = rho^ / (eps0 k^2), E^ = -i k
//             phi^, Nyquist derivatives zeroed, Parseval field energy,
//             tracked mode), inverse FFTs along y of phi^ and Ey^; Ex comes
//             from the inverse of phi^ times -i kx (kx is constant along a
//             column), written column-major Tx[kx][y], Ty[kx][y];
//   rows_inv  per row y: Z = Ex~ + i Ey~ extended to all nx modes by
//             Hermitian symmetry (imaginary parts at kx = 0 and nx/2
//             dropped, as a complex-to-real transform does), one inverse
//             complex FFT, Ex = Re z, Ey = Im z; one block more folds the
//             step's diagnostics.
// The columns also clear the density for the next deposit.
//
// The same launches serve an ensemble's runs of one grid size (blockIdx.y
// picks the run from the run table) and, in their adjoint mode, the
// adjoint's transposed solve psi = S^T g (rows of gx + i gy forward, two
// forward column transforms, the transposed k-space operator and one
// inverse per column, two psi rows per inverse row transform).
//
// The arithmetic per mode is the k-space kernel's (pic_field_dev.cuh); the
// transforms are pic_fft_dev.cuh's.  Replaces (reference paths inside
// taylorj5/msc-thesis, thesisCode/collisionless/double/src/):
//   fourier.cc:15-126 fftPoissonSolver, grid.cc:85-96 computeElectricField.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <vector>

#include "pic_spectral_dev.cuh"

namespace pic {

// LGX: log2 nx.  Block: `pairs` transforms, nx/EL threads each: a pair of
// density rows, or with ADJ one row of the two gradient planes (gx + i gy).
template <int LGX, int EL, bool ADJ>
__global__ void __launch_bounds__(256) spec_rows_fwd_kernel(SpecArgs P)
{
    const SpecArgs A = block_args(P);
    using L = fft::Line<LGX, EL>;
    constexpr int NX = 1 << LGX, TP = L::TP;
    extern __shared__ float2 smem[];
    __shared__ unsigned long long s_q[32];
    const int f = threadIdx.x / TP, t = threadIdx.x - f * TP;
    float2 *buf[1] = {smem + f * A.sa};
    float2 v[1][EL];
    unsigned long long qs = 0;
    if (!A.late) pdl_wait();
    pdl_trigger();
    if (ADJ) {
        const size_t r0 = (size_t)(blockIdx.x * A.pairs + f) * NX;
#pragma unroll
        for (int k = 0; k < EL; ++k)
            v[0][k] = make_float2(A.gx[r0 + L::in(k, t)], A.gy[r0 + L::in(k, t)]);
    } else {
        // all loads first (the density is read-only here), then the
        // conversions and the float density's stores
        const size_t r0 = (size_t)(blockIdx.x * A.pairs + f) * 2 * NX;
        unsigned long long a[EL], b[EL];
#pragma unroll
        for (int k = 0; k < EL; ++k) {
            a[k] = __ldcg(A.rho_fix + r0 + L::in(k, t));
            b[k] = __ldcg(A.rho_fix + r0 + NX + L::in(k, t));
        }
#pragma unroll
        for (int k = 0; k < EL; ++k) {
            qs += a[k] + b[k];
            const float fa = fixed_to_float(a[k], A.mean_fix, A.scale);
            const float fb = fixed_to_float(b[k], A.mean_fix, A.scale);
            A.rho[r0 + L::in(k, t)] = fa;
            A.rho[r0 + NX + L::in(k, t)] = fb;
            v[0][k] = make_float2(fa, fb);
        }
    }
    L::template run<false, 1>(v, buf, t, A.twx);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < EL; ++k) buf[0][L::slot(L::out(k, t))] = v[0][k];
    __syncthreads();
    // split each transform's spectrum; (mode, transform) with the transform
    // fastest, so that the block's rows of one mode are written together
    const int lg = 31 - __clz(A.pairs), np = A.pairs;  // a power of two
    for (int w = threadIdx.x; w < A.nh * np; w += blockDim.x) {
        const int ff = w & (np - 1), k = w >> lg;
        const float2 *bb = smem + ff * A.sa;
        const float2 z = bb[L::slot(k)], m = bb[L::slot((NX - k) & (NX - 1))];
        const float2 ra = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
        const float2 rb = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
        if (ADJ) {
            const size_t i = (size_t)k * A.ny + blockIdx.x * np + ff;
            A.S[i] = ra;
            A.Sy[i] = rb;
        } else {
            const int yy = (blockIdx.x * np + ff) * 2;
            *reinterpret_cast<float4 *>(A.S + (size_t)k * A.ny + yy) = make_float4(ra.x, ra.y, rb.x, rb.y);
        }
    }
    if (!ADJ) {
        qs = block_sum(qs, s_q);
        if (threadIdx.x == 0) atomicAdd(&A.dev->q[acc_slot()], qs);
    }
    if (A.late) pdl_wait();
}

// LGY: log2 ny.  Block: `cols` columns, ny/16 threads each; two buffers per
// column (phi^, then Ey^).
template <int LGY, int EL, bool ADJ>
__global__ void __launch_bounds__(256, 2) spec_cols_kernel(SpecArgs P)
{
    const SpecArgs A = block_args(P);
    using L = fft::Line<LGY, EL>;
    constexpr int NY = 1 << LGY, TP = L::TP;
    extern __shared__ float2 smem[];
    __shared__ double s_fe[32];
    const int c = threadIdx.x / TP, t = threadIdx.x - c * TP;
    const int mx = blockIdx.x * A.cols + c;
    const bool on = mx < A.nh;
    float2 *const b0 = smem + (2 * c) * A.sb, *const b1 = b0 + A.sb;
    const size_t col = (size_t)(on ? mx : 0) * NY;
    float fe = 0.f;
    float2 v[1][EL];
    if (!A.late) pdl_wait();
    pdl_trigger();
    if (!ADJ) {
        // the density, converted by the forward rows, cleared for the next
        // deposit (a memset of its own before; figures at pdl_wait)
        const int n2 = (A.nx << LGY) >> 1, stride = gridDim.x * blockDim.x;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride)
            reinterpret_cast<ulonglong2 *>(A.rho_fix)[i] = make_ulonglong2(0ull, 0ull);
    } else {
        // the scatter planes, transformed by the forward rows, likewise
        const int n4 = (A.nx << LGY) >> 2, stride = gridDim.x * blockDim.x;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
            reinterpret_cast<float4 *>(A.gx)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            reinterpret_cast<float4 *>(A.gy)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    // forward transform of column `src` along y, left in natural order in `bs`
    auto forward = [&](const float2 *src, float2 *bs) {
        float2 *buf[1] = {bs};
#pragma unroll
        for (int k = 0; k < EL; ++k)
            v[0][k] = on ? __ldcg(src + col + L::in(k, t)) : make_float2(0.f, 0.f);
        L::template run<false, 1>(v, buf, t, A.twy);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < EL; ++k) bs[L::slot(L::out(k, t))] = v[0][k];
        __syncthreads();
    };
    forward(A.S, b0);
    if (ADJ) {
        // psi^ = i (kx g^x + ky g^y) / (eps0 N k^2) per mode, inverse along y
        forward(A.Sy, b1);
#pragma unroll
        for (int k = 0; k < EL; ++k) {
            const int my = L::in(k, t);
            v[0][k] = adj_mode(b0[L::slot(my)], b1[L::slot(my)], mx, my, A.nx, NY, A.kx1, A.ky1,
                               A.inv_eps0_n, mx == 0 && my == 0);
        }
        float2 *buf[1] = {b0};
        L::template run<true, 1>(v, buf, t, A.twy);
        if (on) {
#pragma unroll
            for (int k = 0; k < EL; ++k) A.Tx[col + L::out(k, t)] = v[0][k];
        }
        return;
    }
    // k-space: phi^ stays in registers, Ey^ goes to the second buffer; the
    // two inverse transforms run one after the other
#pragma unroll
    for (int k = 0; k < EL; ++k) {
        const int my = L::in(k, t);
        const float2 r = b0[L::slot(my)];
        const KMode K = kspace_mode(r, mx, my, A.nx, NY, A.kx1, A.ky1, A.inv_eps0_n,
                                    mx == 0 && my == 0);
        if (on && mx == A.tmx && my == A.tmy)
            A.dev->mode_amp = sqrt((double)r.x * r.x + (double)r.y * r.y) / ((double)A.nx * NY);
        v[0][k] = K.ph;
        b1[L::slot(my)] = K.ey;
        fe += on ? K.fe : 0.f;
    }
    // the two inverse transforms share one copy of the code: s = 0 turns
    // phi^ (registers, first buffer) into Ex~ = -i kx phi~ (Nyquist kx
    // zeroed), s = 1 turns Ey^ (second buffer) into Ey~
    const float kxe = (2 * mx == A.nx) ? 0.f : A.kx1 * (float)mx;
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
        float2 *const bs = s ? b1 : b0;
        if (s) {
            __syncthreads();  // Ey^ in the second buffer is complete
#pragma unroll
            for (int k = 0; k < EL; ++k) v[0][k] = b1[L::slot(L::in(k, t))];
        }
        float2 *buf[1] = {bs};
        L::template run<true, 1>(v, buf, t, A.twy);
        if (on) {
            float2 *const out = (s ? A.Ty : A.Tx) + col;
#pragma unroll
            for (int k = 0; k < EL; ++k) {
                const float2 u = v[0][k];
                out[L::out(k, t)] = s ? u : make_float2(kxe * u.y, -kxe * u.x);
            }
        }
    }
    const double sum = block_sum((double)fe, s_fe);
    if (threadIdx.x == 0) atomicAdd(&A.dev->fe[acc_slot()], sum);
    if (A.late) pdl_wait();
}

// LGX: log2 nx.  Block: `rows` transforms, nx/16 threads each: row y of Ex~
// and Ey~ into Ex and Ey, or rows 2y and 2y + 1 of psi~ into psi.  With
// A.adv one block more than the rows need folds the step's diagnostics into
// the history beside them (the push's, rows' and columns' sums are complete
// here; a launch of its own before; figures at pdl_wait).
template <int LGX, int EL>
__global__ void __launch_bounds__(256) spec_rows_inv_kernel(SpecArgs P)
{
    const SpecArgs A = block_args(P);
    using L = fft::Line<LGX, EL>;
    constexpr int NX = 1 << LGX, TP = L::TP, HALF = NX >> 1;
    extern __shared__ float2 smem[];
    const int f = threadIdx.x / TP, t = threadIdx.x - f * TP;
    const int nr = A.rows, lg = 31 - __clz(nr);  // a power of two
    const int y0 = blockIdx.x * nr;
    if (!A.late) pdl_wait();
    pdl_trigger();
    if (A.adv && blockIdx.x == gridDim.x - 1) {
        const int lanes = min((int)blockDim.x, 32);  // a power of two
        if ((int)threadIdx.x < lanes)
            advance_state(A.dev, A.hist, A.hist_cap, A.adv, A.fe_scale, lanes);
        if (A.late) pdl_wait();
        return;
    }
    // (mode, row) with the row fastest: the block's rows of one mode are
    // adjacent in Tx and Ty.  nh nr = (EL/2 + EL/nx) times the block's
    // threads: at most EL/2 + 1 items per thread, all loads issued before the
    // shared-memory stores
    constexpr int ITEMS = EL / 2 + 1;
    const int total = (HALF + 1) * nr;
    float2 X[ITEMS], Y[ITEMS];
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const int w = threadIdx.x + q * blockDim.x;
        if (w < total) {
            const size_t i = (size_t)(w >> lg) * A.ny + (size_t)(y0 + (w & (nr - 1))) * A.ys;
            X[q] = __ldcg(A.Tx + i);
            Y[q] = __ldcg(A.Ty + i + A.yo);
        }
    }
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const int w = threadIdx.x + q * blockDim.x;
        if (w < total) {
            const int ff = w & (nr - 1), k = w >> lg;
            float2 x = X[q], y = Y[q];
            if (k == 0 || k == HALF) x.y = y.y = 0.f;
            float2 *bb = smem + ff * A.sc;
            bb[L::slot(k)] = make_float2(x.x - y.y, x.y + y.x);
            if (k > 0 && k < HALF) bb[L::slot(NX - k)] = make_float2(x.x + y.y, y.x - x.y);
        }
    }
    __syncthreads();
    float2 v[1][EL];
    float2 *buf[1] = {smem + f * A.sc};
#pragma unroll
    for (int k = 0; k < EL; ++k) v[0][k] = buf[0][L::slot(L::in(k, t))];
    L::template run<true, 1>(v, buf, t, A.twx);
    const size_t rx = (size_t)(y0 + f) * A.ys * NX, ry = rx + (size_t)A.yo * NX;
#pragma unroll
    for (int k = 0; k < EL; ++k) {
        const int i = L::out(k, t);
        A.ex[rx + i] = v[0][k].x;
        A.ey[ry + i] = v[0][k].y;
    }
    if (A.late) pdl_wait();
}

static int pow2_floor(int n)
{
    int p = 1;
    while (2 * p <= n) p *= 2;
    return p;
}

static int ilog2(int n)
{
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

bool spectral_size_ok(int nx, int ny)
{
    auto ok = [](int n) { return n >= 16 && n <= 4096 && (n & (n - 1)) == 0; };
    return ok(nx) && ok(ny);
}

bool spectral_wanted(int nx, int ny)
{
    const char *solver = getenv("PIC_FIELD_SOLVER");
    return spectral_size_ok(nx, ny) && !(solver && strcmp(solver, "cufft") == 0);
}

// the transforms' per-pass twiddle tables (fft::twiddle_len entries for nx,
// then for ny): pass (lgns, lgr) with lgns > 0 holds W_(Ns R)^(r m) at
// r Ns + m, r < R, m < Ns
static void append_twiddles(std::vector<float2> &t, int lgn)
{
    const double pi = 3.14159265358979323846;
    for (int lgns = 0; lgns < lgn; lgns += fft::pass_lgr(lgn, lgns)) {
        if (lgns == 0) continue;
        const int R = 1 << fft::pass_lgr(lgn, lgns), Ns = 1 << lgns;
        for (int r = 0; r < R; ++r)
            for (int m = 0; m < Ns; ++m) {
                const double a = 2.0 * pi * (double)(r * m) / (double)(Ns * R);
                t.push_back(make_float2((float)std::cos(a), (float)-std::sin(a)));
            }
    }
}

pic_status spectral_twiddles(int nx, int ny, float2 **tw)
{
    std::vector<float2> t;
    append_twiddles(t, ilog2(nx));
    append_twiddles(t, ilog2(ny));
    t.push_back(make_float2(1.f, 0.f));  // never empty (16-point transforms need none)
    PIC_CUDA(cudaMalloc(tw, t.size() * sizeof(float2)));
    PIC_CUDA(cudaMemcpy(*tw, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice));
    return PIC_OK;
}

// The solve of `batch` runs of one grid size (L.A.runs set) or one run: the
// field solve, or with adj the adjoint solve (A.gx, A.gy -> psi in A.ex).  The
// field solve leaves the fixed-point density cleared.
static pic_status plan_kernels(SpecLaunch &L, int batch, bool adj = false)
{
    SpecArgs &A = L.A;
    const int nx = A.nx, ny = A.ny, nh = A.nh;
    A.lgx = ilog2(nx);
    A.lgy = ilog2(ny);
    A.twy = A.twx + fft::twiddle_len(A.lgx);
    A.ys = adj ? 2 : 1;
    A.yo = adj ? 1 : 0;
    if (!adj && batch >= 1 && plan_small(L, A.lgx, A.lgy, batch)) return PIC_OK;
    // Elements per thread: 16, or 4 where the grids leave the GPU to the latency
    // of one thread's chain.  Step on single handles (23 particles per cell, 16
    // and 4): 128x512 38.4 and 29.5 us, 256^2 35.2 and 28.8, 512^2 80.2 and 72.9,
    // 1024x512 131.3 and 128.0, 1024^2 228.6 and 235.2; ensembles (16 per cell):
    // two 256^2 runs 44.4 and 38.4, eight 116.5 and 114.4, 32 352 and 358; two
    // 512^2 runs 125.6 and 124.6, four 216.6 and 220.8.  The field keeps its
    // bits; the adjoint's psi^ goes from its operator straight into the transform
    // and does not (a chaotic run's gradients three times as far off as by the
    // order of their sums), so that solve stays at 16.
    const bool quads = !adj && (long long)nx * ny * batch <= 524288;
    auto elements = [&](int lg) { return quads && lg >= 7 && lg <= 10 ? 4 : 16; };
    const int ex = elements(A.lgx), ey = elements(A.lgy);
    const int tpx = nx / ex, tpy = ny / ey;
    // transforms of the forward and the inverse rows: row pairs and rows
    // (field), rows and row pairs (adjoint)
    const int na = adj ? ny : ny / 2, nc = adj ? ny / 2 : ny;
    // transforms per block: at most 256 threads, and no more than spreads the
    // batch's transforms over about one block per SM (small grids otherwise
    // run on a few SMs), but at least a warp's worth where the grid allows
    const int sms = device_sms();
    auto per_block = [&](int tp, int items) {
        const int spread = (int)std::max(1ll, (long long)items * batch / sms);
        int k = std::min(256 / tp, pow2_floor(spread));
        k = std::max(k, std::min(32 / tp, items));
        return std::max(1, std::min(k, items));
    };
    A.pairs = per_block(tpx, na);
    A.cols = per_block(tpy, nh);
    A.rows = per_block(tpx, nc);
    // interleaved buffers read by consecutive lanes start on different banks
    auto stride = [](int n, int el, int extra) {
        return el == 4 ? n + n / 4 + extra : fft::buf_stride(n, extra);
    };
    A.sa = stride(nx, ex, 16 / std::min(A.pairs, 16));
    A.sb = stride(ny, ey, 8);
    A.sc = stride(nx, ex, 16 / std::min(A.rows, 16));
    const size_t ma = (size_t)A.pairs * A.sa * sizeof(float2);
    const size_t mb = (size_t)2 * A.cols * A.sb * sizeof(float2);
    const size_t mc = (size_t)A.rows * A.sc * sizeof(float2);
    const void *ka = nullptr, *kb = nullptr, *kc = nullptr;
    switch (A.lgx * 32 + ex) {
#define PIC_SPEC_X(L, EL)                                                                      \
    case L * 32 + EL:                                                                          \
        ka = adj ? (const void *)spec_rows_fwd_kernel<L, 16, true>                             \
                 : (const void *)spec_rows_fwd_kernel<L, EL, false>;                           \
        kc = (const void *)spec_rows_inv_kernel<L, EL>;                                        \
        break;
        PIC_SPEC_X(4, 16) PIC_SPEC_X(5, 16) PIC_SPEC_X(6, 16) PIC_SPEC_X(7, 16) PIC_SPEC_X(8, 16)
        PIC_SPEC_X(9, 16) PIC_SPEC_X(10, 16) PIC_SPEC_X(11, 16) PIC_SPEC_X(12, 16)
        PIC_SPEC_X(7, 4) PIC_SPEC_X(8, 4) PIC_SPEC_X(9, 4) PIC_SPEC_X(10, 4)
#undef PIC_SPEC_X
    }
    switch (A.lgy * 32 + ey) {
#define PIC_SPEC_Y(L, EL)                                                                      \
    case L * 32 + EL:                                                                          \
        kb = adj ? (const void *)spec_cols_kernel<L, 16, true>                                 \
                 : (const void *)spec_cols_kernel<L, EL, false>;                               \
        break;
        PIC_SPEC_Y(4, 16) PIC_SPEC_Y(5, 16) PIC_SPEC_Y(6, 16) PIC_SPEC_Y(7, 16) PIC_SPEC_Y(8, 16)
        PIC_SPEC_Y(9, 16) PIC_SPEC_Y(10, 16) PIC_SPEC_Y(11, 16) PIC_SPEC_Y(12, 16)
        PIC_SPEC_Y(7, 4) PIC_SPEC_Y(8, 4) PIC_SPEC_Y(9, 4) PIC_SPEC_Y(10, 4)
#undef PIC_SPEC_Y
    }
    if (!ka || !kb || batch < 1) {
        set_error("spectral solve: grid side outside 16..4096");
        return PIC_ERR_INVALID_ARG;
    }
    PIC_TRY(allow_dynamic_smem(ka, ma));
    PIC_TRY(allow_dynamic_smem(kb, mb));
    PIC_TRY(allow_dynamic_smem(kc, mc));
    const unsigned nb = (unsigned)batch;
    const unsigned fold = A.adv ? 1u : 0u;
    L.kernel[0] = ka, L.kernel[1] = kb, L.kernel[2] = kc;
    L.smem[0] = ma, L.smem[1] = mb, L.smem[2] = mc;
    L.grid[0] = dim3(na / A.pairs, nb), L.block[0] = dim3(A.pairs * tpx);
    L.grid[1] = dim3((nh + A.cols - 1) / A.cols, nb), L.block[1] = dim3(A.cols * tpy);
    L.grid[2] = dim3(nc / A.rows + fold, nb), L.block[2] = dim3(A.rows * tpx);
    return PIC_OK;
}

// Stage by stage over independent solves, which overlap within a stage (the
// grid sizes of an ensemble: 8 runs of three sizes, 10 M particles, 103 -> 83 us
// a step; 16 of four, 209 M, 1571 -> 1542).
static pic_status launch_kernels(SpecLaunch *L, size_t count, cudaStream_t st)
{
    for (int k = 0; k < 3; ++k) {
        int late = 0;
        for (size_t i = 0; i < count; ++i) {
            if (!L[i].kernel[k]) continue;
            L[i].A.late = late;
            late = 1;
            void *args[] = {&L[i].A};
            PIC_TRY(launch_dependent(L[i].kernel[k], L[i].grid[k], L[i].block[k], L[i].smem[k], st, args));
        }
    }
    return PIC_OK;
}

void spectral_args(pic_handle *h, int adv, float *e, SpecArgs &A)
{
    const Geometry &g = h->g;
    memset(&A, 0, sizeof A);
    A.rho_fix = h->rho_fix;
    A.rho = h->rho;
    A.S = h->rhohat;
    A.Tx = h->ehat;
    A.Ty = h->ehat + (size_t)g.nh * g.ny;
    A.ex = e ? e : h->e;
    A.ey = A.ex + (size_t)g.nx * g.ny;
    A.nx = g.nx;
    A.ny = g.ny;
    A.nh = g.nh;
    A.twx = h->tw;
    A.mean_fix = h->mean_fix;
    A.scale = (float)(h->q_unit / (4294967296.0 * g.dx * g.dy));
    A.kx1 = (float)(2.0 * 3.14159265358979323846 / g.Lx);
    A.ky1 = (float)(2.0 * 3.14159265358979323846 / g.Ly);
    A.inv_eps0_n = (float)(1.0 / (h->cfg.eps0 * (double)g.nx * (double)g.ny));
    A.tmx = h->track_mx;
    A.tmy = h->track_my;
    A.dev = h->dev;
    A.hist = h->hist;
    A.hist_cap = h->hist_cap;
    A.adv = adv;
    A.fe_scale = 0.5 * h->cfg.eps0 * g.dx * g.dy * (double)g.nx * (double)g.ny;
}

pic_status launch_spectral(pic_handle *h, int adv, float *e)
{
    SpecLaunch L;
    spectral_args(h, adv, e, L.A);
    PIC_TRY(plan_kernels(L, 1));
    return launch_kernels(&L, 1, h->stream);
}

pic_status launch_spectral_runs(const EnsRun *runs, const SpecGroup *groups, int ngroups,
                                unsigned long long *rho_fix, float *rho, float2 *rhohat,
                                float2 *ehat, float *e, DevState *devs, double *hist, int hist_cap,
                                int adv, cudaStream_t st)
{
    std::vector<SpecLaunch> L;
    for (int i = 0; i < ngroups; ++i) {
        const SpecGroup &G = groups[i];
        // a grid's y dimension holds at most 65535 runs
        for (int b = 0; b < G.count; b += 65535) {
            L.emplace_back();
            SpecArgs &A = L.back().A;
            memset(&A, 0, sizeof A);
            A.rho_fix = rho_fix;
            A.rho = rho;
            A.S = rhohat;
            A.Tx = ehat;
            A.ex = e;
            A.nx = G.nx;
            A.ny = G.ny;
            A.nh = G.nx / 2 + 1;
            A.twx = G.tw;
            A.tmx = A.tmy = -1;
            A.dev = devs;
            A.hist = hist;
            A.hist_cap = hist_cap;
            A.adv = adv;
            A.runs = runs;
            A.first = G.first + b;
            PIC_TRY(plan_kernels(L.back(), std::min(65535, G.count - b)));
        }
    }
    return launch_kernels(L.data(), L.size(), st);
}

// psi = S^T g on a power-of-two handle: gx, gy (ncell each) -> psi; gh
// (2 ny nh) and ph (ny nh) are scratch
pic_status launch_spectral_adjoint(pic_handle *h, float *gx, float *gy, float2 *gh, float2 *ph,
                                   float *psi)
{
    const Geometry &g = h->g;
    SpecLaunch L;
    SpecArgs &A = L.A;
    memset(&A, 0, sizeof A);
    A.gx = gx;
    A.gy = gy;
    A.S = gh;
    A.Sy = gh + (size_t)g.nh * g.ny;
    A.Tx = A.Ty = ph;
    A.ex = A.ey = psi;
    A.nx = g.nx;
    A.ny = g.ny;
    A.nh = g.nh;
    A.twx = h->tw;
    A.kx1 = (float)(2.0 * 3.14159265358979323846 / g.Lx);
    A.ky1 = (float)(2.0 * 3.14159265358979323846 / g.Ly);
    A.inv_eps0_n = (float)(1.0 / (h->cfg.eps0 * (double)g.nx * (double)g.ny));
    A.tmx = A.tmy = -1;
    A.dev = h->dev;
    PIC_TRY(plan_kernels(L, 1, true));
    return launch_kernels(&L, 1, h->stream);
}

}  // namespace pic
