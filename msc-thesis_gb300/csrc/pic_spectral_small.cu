// pic_spectral_small.cu -- the spectral field solve of small grids (power-of-two
// sides 32..128) in one kernel: one cluster of eight blocks per run.
//
// On these grids each of the three kernels of pic_spectral.cu is a few blocks
// of a warp or two, bound by its launch and by the latency of one thread's
// radix-16 chain.  Here the blocks of a cluster split the rows, then the
// columns, then the rows again, and hand the transposed spectra to each other
// through distributed shared memory:
//   rows     block r transforms its row pairs (as spec_rows_fwd_kernel) and
//            writes each mode to the block that owns its column
//   columns  forward, k-space operator, two inverses (as spec_cols_kernel);
//            each value goes to the block that owns its row
//   rows     inverse (as spec_rows_inv_kernel) into Ex, Ey
// with a cluster barrier between the stages.  A thread holds four elements
// so that a transform lies within a warp and needs no block
// barrier, and its chain is a quarter as long.  Global writes wait
// until the last barrier, which would otherwise wait for them; the sums of
// charge and field energy go to the last block through shared memory as well,
// whose extra warp does the diagnostics fold beside the inverse rows.
// One step of 64^2 cells with 16 particles each: 20.5 -> 12.0 us, of 128^2 with
// 100 each: 34.2 -> 27.1 us; eight runs of small grids in one ensemble: 87 ->
// 79 us.  The results keep their bits.  The same split with the three kernels'
// radix-16 transforms, block barriers, global sums and the fold by atomics:
// 17.5, 31.9 and 93 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "pic_spectral_dev.cuh"

namespace pic {
namespace {

constexpr int E4 = 4;  // elements per thread

constexpr int max_of(int a, int b) { return a > b ? a : b; }
constexpr int warps_of(int threads) { return (threads + 31) / 32; }

// Work split and shared memory (float2 slots) of a block.
template <int LGX, int LGY>
struct Small {
    static constexpr int NX = 1 << LGX, NY = 1 << LGY, NH = NX / 2 + 1;
    static constexpr int TPX = NX / E4, TPY = NY / E4;  // threads per transform (8..32)
    static constexpr int NP = NY / 2 / CL;              // row pairs of a block
    static constexpr int NR = NY / CL;                  // rows
    static constexpr int NC = (NH + CL - 1) / CL;       // columns
    static constexpr int WP = warps_of(NP * TPX), WC = warps_of(NC * TPY), WR = warps_of(NR * TPX);
    static constexpr int WARPS = max_of(WC, WR), T = 32 * (WARPS + 1);  // and the fold's warp
    static_assert(NR * TPX == 32 * WR && WP <= WR, "block shape");
    static constexpr int SX = fft::buf_stride(NX, 2), SY = fft::buf_stride(NY, 2);
    static constexpr int WORK =
        max_of(max_of(WP, WR) * (32 / TPX) * SX, 2 * WC * (32 / TPY) * SY);
    static constexpr int COLS = NC * NY;                // spectra of the block's columns
    static constexpr int ROWS = NR * NH;                // Ex~ (and Ey~) of its rows
    static constexpr size_t BYTES = sizeof(float2) * (WORK + COLS + 2 * ROWS);
    static_assert(WORK % 2 == 0, "the columns start on 16 bytes");
};

// A thread's part in transforms of length 2^LGN (32 <= n <= 128) on n/4
// threads of a warp: the radix-16 pass and the radix-2, 4 or 8 pass of
// fft::transform in the same order of operations, split over the four (and
// two) threads that share a butterfly, so that every result keeps its bits.
template <int LGN>
struct Part {
    static constexpr int N = 1 << LGN, TP = N / E4, Q = N / 16;
    int t;
    float c1, s1, c2, s2;  // W_16^j and W_16^2j, j = t / Q: this thread's lane of its butterfly
    float2 tw[E4];         // second pass: the factor of element t + k TP

    __device__ __forceinline__ Part(int t, const float2 *__restrict__ tab) : t(t)
    {
        const float C = 0.92387953251128675613f;  // cos(pi / 8)
        const float S = 0.38268343236508977173f;  // sin(pi / 8)
        const float H = 0.70710678118654752440f;  // sqrt(1 / 2)
        const int j = t / Q;
        c1 = j == 0 ? 1.f : j == 1 ? C : j == 2 ? H : S;
        s1 = j == 0 ? 0.f : j == 1 ? S : j == 2 ? H : C;
        c2 = j == 0 ? 1.f : j == 1 ? H : j == 2 ? 0.f : -H;
        s2 = j == 0 ? 0.f : j == 2 ? 1.f : H;
#pragma unroll
        for (int k = 0; k < E4; ++k) tw[k] = __ldg(tab + t + k * TP);  // entry 16 r + m = the element
    }

    // element index of register k after run(): natural but for n = 128
    __device__ __forceinline__ int index(int k) const
    {
        return LGN == 7 ? (t & 15) + 64 * (t >> 4) + 16 * fft::rev2(k) : t + k * TP;
    }

    // v[a][k] holds element t + k TP on entry, element index(k) on exit
    template <bool INV, int NA>
    __device__ __forceinline__ void run(float2 (&v)[NA][E4], float2 *const (&buf)[NA]) const
    {
        const int j = t / Q, o = 17 * (t % Q);  // slot pad(16 t0 + r) = 17 t0 + r
        // radix 16, outputs 4 g + j' of stages h = 8 and 4 in register g
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            fft::far_pairs<INV>(v[a], c1, s1, -s1, c1);
            fft::near_pairs<INV>(v[a], c2, s2);
        }
        __syncwarp();  // every thread has read the previous contents
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int g = 0; g < E4; ++g) {
                // registers 1 and 2 hold positions j + 4 and j + 8
                buf[a][o + 4 * g + j] = v[a][g];
            }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; ++a) {
#pragma unroll
            for (int i = 0; i < E4; ++i) v[a][i] = buf[a][o + 4 * j + i];
            // stages h = 2 and 1
            fft::far_pairs<INV>(v[a], 1.f, 0.f, 0.f, 1.f);
            fft::near_pairs<INV>(v[a], 1.f, 0.f);
        }
        __syncwarp();
        // position 4 j + i is output 4 fft::rev2(i) + fft::rev2(j)
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int i = 0; i < E4; ++i) buf[a][o + 4 * fft::rev2(i) + fft::rev2(j)] = v[a][i];
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; ++a) {
#pragma unroll
            for (int k = 0; k < E4; ++k) {
                v[a][k] = buf[a][fft::pad(t + k * TP)];
                if (LGN == 7 || k * TP >= 16) {  // the factor is 1 below element 16
                    float2 w = tw[k];
                    if (INV) w.y = -w.y;
                    v[a][k] = fft::cmul(v[a][k], w);
                }
            }
            if (LGN == 5) {
                fft::far_pairs<INV>(v[a], 1.f, 0.f, 1.f, 0.f);
            } else if (LGN == 6) {
                fft::dft<4, INV>(v[a]);
            } else {
                // register k is input r = q + 2 k of a radix-8 butterfly; stages
                // h = 4 and 2, then h = 1 with the thread of the other q
                const float H = 0.70710678118654752440f;
                const bool q = t & 16;
                fft::far_pairs<INV>(v[a], q ? H : 1.f, q ? H : 0.f, q ? -H : 0.f, q ? H : 1.f);
                fft::near_pairs<INV>(v[a], q ? 0.f : 1.f, q ? 1.f : 0.f);
#pragma unroll
                for (int k = 0; k < E4; ++k) {
                    const float2 z = make_float2(__shfl_xor_sync(~0u, v[a][k].x, 16),
                                                 __shfl_xor_sync(~0u, v[a][k].y, 16));
                    v[a][k] = q ? fft::csub(z, v[a][k]) : fft::cadd(v[a][k], z);
                }
            }
        }
    }
};

template <int LGX, int LGY>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(Small<LGX, LGY>::T)
spec_small_kernel(SpecArgs P)
{
    using Z = Small<LGX, LGY>;
    extern __shared__ __align__(16) float2 smem[];
    __shared__ unsigned long long s_q[CL * Z::WP];
    __shared__ double s_fe[CL * Z::WC];
    __shared__ double s_amp;
    const SpecArgs A = block_args(P);
    const unsigned rank = cluster_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float2 *const work = smem, *const cols = work + Z::WORK;
    float2 *const rowx = cols + Z::COLS, *const rowy = rowx + Z::ROWS;
    const bool tracked = A.tmx >= 0 && A.tmx < Z::NH && A.tmy >= 0 && A.tmy < Z::NY;
    const Part<LGX> fx(threadIdx.x % Z::TPX, A.twx);
    const Part<LGY> fy(threadIdx.x % Z::TPY, A.twy);
    cluster_arrive();  // the cluster's blocks run
    if (!A.late) pdl_wait();
    pdl_trigger();

    // ---- row pairs along x
    float fa[E4], fb[E4];
    const int fp = threadIdx.x / Z::TPX, tp = threadIdx.x % Z::TPX;
    const bool onp = fp < Z::NP;
    const size_t r0 = (size_t)(rank * Z::NP + fp) * 2 * Z::NX;
    unsigned long long a[E4], b[E4];
    if (onp) {
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            a[k] = __ldcg(A.rho_fix + r0 + tp + k * Z::TPX);
            b[k] = __ldcg(A.rho_fix + r0 + Z::NX + tp + k * Z::TPX);
        }
    }
    cluster_wait();
    if (warp < Z::WP) {
        float2 v[1][E4];
        unsigned long long qs = 0;
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            if (onp) {
                qs += a[k] + b[k];
                fa[k] = fixed_to_float(a[k], A.mean_fix, A.scale);
                fb[k] = fixed_to_float(b[k], A.mean_fix, A.scale);
            } else {
                fa[k] = fb[k] = 0.f;
            }
            v[0][k] = make_float2(fa[k], fb[k]);
        }
        float2 *buf[1] = {work + fp * Z::SX};
        fx.template run<false>(v, buf);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < E4; ++k) buf[0][fft::pad(fx.index(k))] = v[0][k];
        __syncwarp();
        if (onp) {
#pragma unroll
            for (int k = tp; k < Z::NH; k += Z::TPX) {
                const float2 z = buf[0][fft::pad(k)], m = buf[0][fft::pad((Z::NX - k) & (Z::NX - 1))];
                const float2 ra = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
                const float2 rb = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
                const int c = k / Z::NC;
                put4(remote(cols + (k - c * Z::NC) * Z::NY + ((int)rank * Z::NP + fp) * 2, c), ra, rb);
            }
        }
        qs = warp_sum(qs);
        if (lane == 0) put(remote(s_q + rank * Z::WP + warp, CL - 1), qs);
    }
    cluster_arrive();
    cluster_wait();

    // ---- columns along y
    if (warp < Z::WC) {
        constexpr int TP = Z::TPY;
        const int c = threadIdx.x / TP, t = threadIdx.x % TP;
        const int mx = (int)rank * Z::NC + c;
        const bool on = c < Z::NC && mx < Z::NH;
        float2 *const b0 = work + 2 * c * Z::SY, *const b1 = b0 + Z::SY;
        float2 u[2][E4];
        float fe = 0.f;
        {
            float2 v[1][E4];
            float2 *buf[1] = {b0};
#pragma unroll
            for (int k = 0; k < E4; ++k)
                v[0][k] = on ? cols[c * Z::NY + t + k * TP] : make_float2(0.f, 0.f);
            fy.template run<false>(v, buf);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < E4; ++k) {
                const int my = fy.index(k);
                const KMode K = kspace_mode(v[0][k], mx, my, Z::NX, Z::NY, A.kx1, A.ky1, A.inv_eps0_n,
                                            mx == 0 && my == 0);
                b0[fft::pad(my)] = K.ph;
                b1[fft::pad(my)] = K.ey;
                fe += on ? K.fe : 0.f;
                if (tracked && on && mx == A.tmx && my == A.tmy) {
                    const double x = v[0][k].x, y = v[0][k].y;
                    const double amp = sqrt(x * x + y * y) / ((double)Z::NX * Z::NY);
                    put(remote(&s_amp, CL - 1), (unsigned long long)__double_as_longlong(amp));
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            u[0][k] = b0[fft::pad(t + k * TP)];
            u[1][k] = b1[fft::pad(t + k * TP)];
        }
        const float kxe = (2 * mx == Z::NX) ? 0.f : A.kx1 * (float)mx;
        float2 *buf[2] = {b0, b1};
        fy.template run<true>(u, buf);
        if (on) {
#pragma unroll
            for (int k = 0; k < E4; ++k) {
                const int y = fy.index(k), o = (y % Z::NR) * Z::NH + mx;
                put2(remote(rowx + o, y / Z::NR), make_float2(kxe * u[0][k].y, -kxe * u[0][k].x));
                put2(remote(rowy + o, y / Z::NR), u[1][k]);
            }
        }
        const double sum = warp_sum((double)fe);
        if (lane == 0)
            put(remote(s_fe + rank * Z::WC + warp, CL - 1), (unsigned long long)__double_as_longlong(sum));
    }
    cluster_arrive();
    cluster_wait();

    // ---- rows back
    if (warp < Z::WR) {
        constexpr int TP = Z::TPX, HALF = Z::NX / 2;
        const int f = threadIdx.x / TP, t = threadIdx.x % TP;
        float2 v[1][E4];
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            const int i = t + k * TP, m = i <= HALF ? i : Z::NX - i;
            float2 x = rowx[f * Z::NH + m], y = rowy[f * Z::NH + m];
            if (m == 0 || m == HALF) x.y = y.y = 0.f;
            v[0][k] = i <= HALF ? make_float2(x.x - y.y, x.y + y.x) : make_float2(x.x + y.y, y.x - x.y);
        }
        float2 *buf[1] = {work + f * Z::SX};
        fx.template run<true>(v, buf);
        const size_t r = (size_t)(rank * Z::NR + f) * Z::NX;
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            A.ex[r + fx.index(k)] = v[0][k].x;
            A.ey[r + fx.index(k)] = v[0][k].y;
        }
    } else if (rank == CL - 1 && warp == Z::WARPS) {
        // the solve's sums, then the diagnostics fold (the push's sums are
        // complete since the wait above)
        unsigned long long q = 0;
        double fe = 0.0;
        for (int l = lane; l < CL * Z::WP; l += 32) q += s_q[l];
        for (int l = lane; l < CL * Z::WC; l += 32) fe += s_fe[l];
        if (A.adv & ADV_FIELD) {
            advance_state(A.dev, A.hist, A.hist_cap, A.adv, A.fe_scale, 32, fe, q, tracked ? &s_amp : nullptr);
        } else {
            if (A.adv) advance_state(A.dev, A.hist, A.hist_cap, A.adv, A.fe_scale, 32);
            A.dev->q[lane] = __ldcg(&A.dev->q[lane]) + q;
            A.dev->fe[lane] = __ldcg(&A.dev->fe[lane]) + fe;
            if (tracked && lane == 0) A.dev->mode_amp = s_amp;
        }
    }
    if (onp) {
#pragma unroll
        for (int k = 0; k < E4; ++k) {
            const size_t i = r0 + tp + k * Z::TPX;
            A.rho[i] = fa[k];
            A.rho[i + Z::NX] = fb[k];
            A.rho_fix[i] = 0ull;  // cleared for the next deposit
            A.rho_fix[i + Z::NX] = 0ull;
        }
    }
    if (A.late) pdl_wait();
}

template <int LGX, int LGY>
bool plan(SpecLaunch &L, int batch)
{
    using Z = Small<LGX, LGY>;
    const void *const kernel = (const void *)spec_small_kernel<LGX, LGY>;
    if (allow_dynamic_smem(kernel, Z::BYTES) != PIC_OK) return false;
    L.kernel[0] = kernel;
    L.kernel[1] = L.kernel[2] = nullptr;
    L.grid[0] = dim3(CL, batch);
    L.block[0] = dim3(Z::T);
    L.smem[0] = Z::BYTES;
    return true;
}

}  // namespace

bool plan_small(SpecLaunch &L, int lgx, int lgy, int batch)
{
    switch (16 * lgx + lgy) {
#define PIC_SMALL(X, Y)                                                                        \
    case 16 * X + Y: return plan<X, Y>(L, batch);
        PIC_SMALL(5, 5) PIC_SMALL(5, 6) PIC_SMALL(5, 7)
        PIC_SMALL(6, 5) PIC_SMALL(6, 6) PIC_SMALL(6, 7)
        PIC_SMALL(7, 5) PIC_SMALL(7, 6) PIC_SMALL(7, 7)
#undef PIC_SMALL
    }
    return false;
}

}  // namespace pic
