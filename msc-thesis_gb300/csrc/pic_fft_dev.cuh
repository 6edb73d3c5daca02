// pic_fft_dev.cuh -- shared-memory complex FFTs of power-of-two lengths
// 16..4096 for the spectral Poisson solve (pic_spectral.cu).
//
// Stockham auto-sort passes as published by Govindaraju et al., "High
// performance discrete Fourier transforms on graphics processors" (SC'08):
// pass p with radix R over sub-transforms of length Ns takes butterfly j's
// inputs at j + r N/R, multiplies input r by W_N^(r (j mod Ns) N/(Ns R)),
// transforms the R values and writes output r to
// (j / Ns) Ns R + (j mod Ns) + r Ns; after the last pass the sequence is in
// natural order.  Passes are of radix 16, plus one of radix 8, 4 or 2 for the
// remaining factor.  Every thread of a transform holds 16 elements in
// registers (its butterflies of the pass: j = t + b N/16 for b < 16/R); the
// passes exchange through one shared-memory buffer per transform, indexed
// with one pad slot per 16 elements against bank conflicts.  The length is a
// template parameter, so that all but a per-thread base of every
// shared-memory and twiddle address is a compile-time offset.  Twiddles come
// from per-pass tables computed in double on the host (twiddle_len entries
// per length; a warp reads consecutive entries).
#pragma once
#include <cuda_runtime.h>

namespace pic {
namespace fft {

constexpr int E = 16;  // elements per thread

// shared-memory float2 slots of one transform's buffer; `extra` spreads
// interleaved buffers over the banks
__host__ __device__ constexpr int buf_stride(int n, int extra) { return n + (n >> 4) + extra; }
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// a * exp(-+2 pi i k / 16) for k in [0, 8) (- forward, + inverse); k is a
// compile-time constant after unrolling, so the switch folds away
template <bool INV>
__device__ __forceinline__ float2 w16(float2 a, int k)
{
    const float C = 0.92387953251128675613f;  // cos(pi / 8)
    const float S = 0.38268343236508977173f;  // sin(pi / 8)
    const float H = 0.70710678118654752440f;  // sqrt(1 / 2)
    float c, s;
    switch (k) {
    case 0: return a;
    case 4: return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
    case 1: c = C; s = S; break;
    case 2: c = H; s = H; break;
    case 3: c = S; s = C; break;
    case 5: c = -S; s = C; break;
    case 6: c = -H; s = H; break;
    default: c = -C; s = S; break;
    }
    if (!INV) s = -s;
    return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c));
}

template <int R>
__host__ __device__ constexpr int bit_reverse(int i)
{
    int r = 0;
    for (int m = 1, b = R >> 1; m < R; m <<= 1, b >>= 1)
        if (i & m) r |= b;
    return r;
}

// in-register DFT of v[0, R), natural order in and out: radix-2 decimation
// in frequency (butterfly twiddle W_2h^j = W_16^(16 j / 2h)), then the
// bit-reversal permutation (register renaming)
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 *v)
{
#pragma unroll
    for (int h = R / 2; h >= 1; h >>= 1) {
#pragma unroll
        for (int s = 0; s < R; s += 2 * h) {
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float2 a = v[s + j], b = v[s + j + h];
                v[s + j] = cadd(a, b);
                v[s + j + h] = w16<INV>(csub(a, b), j * (16 / (2 * h)));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = bit_reverse<R>(i);
        if (r > i) {
            const float2 t = v[i];
            v[i] = v[r];
            v[r] = t;
        }
    }
}

// Pass of a length-2^LGN transform over sub-transforms of length 2^LGNS:
// radix 2^LGR, LGR = 4 while four or more bits remain (LGNS is 0, 4 or 8).
template <int LGN, int LGNS>
struct Pass {
    static constexpr int LGR = (LGN - LGNS) >= 4 ? 4 : (LGN - LGNS);
    static constexpr int R = 1 << LGR, NS = 1 << LGNS, TP = 1 << (LGN - 4), NB = E / R;
    static constexpr bool LAST = LGNS + LGR == LGN;
    static constexpr int TWLEN = LGNS > 0 ? R * NS : 0;  // its twiddle table
};

__host__ __device__ constexpr int pass_lgr(int lgn, int lgns) { return (lgn - lgns) >= 4 ? 4 : (lgn - lgns); }
__host__ __device__ inline int twiddle_len(int lgn)
{
    int len = 0;
    for (int lgns = 0; lgns < lgn; lgns += pass_lgr(lgn, lgns))
        if (lgns > 0) len += 1 << (lgns + pass_lgr(lgn, lgns));
    return len;
}

// twiddles and butterflies of one pass; tw is the pass's table, entry
// r Ns + m = W_(Ns R)^(r m): consecutive lanes (consecutive m = j mod Ns) read
// consecutive entries
template <int LGN, int LGNS, bool INV>
__device__ __forceinline__ void pass_compute(float2 (&v)[E], int t, const float2 *__restrict__ tw)
{
    using P = Pass<LGN, LGNS>;
#pragma unroll
    for (int b = 0; b < P::NB; ++b) {
        if (LGNS > 0) {
            const float2 *tb = tw + ((t + b * P::TP) & (P::NS - 1));
#pragma unroll
            for (int r = 1; r < P::R; ++r) {
                float2 w = __ldg(tb + r * P::NS);
                if (INV) w.y = -w.y;
                v[b * P::R + r] = cmul(v[b * P::R + r], w);
            }
        }
        dft<P::R, INV>(v + b * P::R);
    }
}

// Registers of pass (LGN, LGNS): k = b R + r holds input r of butterfly
// j = t + b TP, element j + r N/R.  Where an offset is a multiple of 16,
// pad(x + c) = pad(x) + c + c/16 keeps it a compile-time offset.
template <int LGN, int LGNS, int NA>
__device__ __forceinline__ void load_pass(float2 (&v)[NA][E], float2 *const (&buf)[NA], int t)
{
    using P = Pass<LGN, LGNS>;
    constexpr int STRIDE = (1 << LGN) / P::R;
#pragma unroll
    for (int b = 0; b < P::NB; ++b) {
        const int x = t + b * P::TP, px = pad(x);
#pragma unroll
        for (int r = 0; r < P::R; ++r) {
            const int c = r * STRIDE;
            const int s = (STRIDE % 16 == 0) ? px + c + c / 16 : pad(x + c);
#pragma unroll
            for (int a = 0; a < NA; ++a) v[a][b * P::R + r] = buf[a][s];
        }
    }
}

// outputs of pass (LGN, LGNS): output r of butterfly j to
// (j / Ns) Ns R + (j mod Ns) + r Ns
template <int LGN, int LGNS, int NA>
__device__ __forceinline__ void store_pass(float2 (&v)[NA][E], float2 *const (&buf)[NA], int t)
{
    using P = Pass<LGN, LGNS>;
    static_assert(LGNS != 0 || P::R == 16, "the first pass is of radix 16");
#pragma unroll
    for (int b = 0; b < P::NB; ++b) {
        const int j = t + b * P::TP;
        if constexpr (LGNS == 0) {
            // slot pad(16 j + r) = 17 j + r
#pragma unroll
            for (int r = 0; r < P::R; ++r)
#pragma unroll
                for (int a = 0; a < NA; ++a) buf[a][17 * j + r] = v[a][b * P::R + r];
        } else {
            const int pd = pad(((j >> LGNS) << (LGNS + P::LGR)) + (j & (P::NS - 1)));
#pragma unroll
            for (int r = 0; r < P::R; ++r) {
                const int c = r * P::NS;  // Ns >= 16
#pragma unroll
                for (int a = 0; a < NA; ++a) buf[a][pd + c + c / 16] = v[a][b * P::R + r];
            }
        }
    }
}

// Transforms of length 2^LGN (16 <= n <= 4096), NA of them per thread (one
// buffer each).  On entry v[a][k] holds element t + k n/16 of transform a;
// on exit v[a][k] holds output element result_index<LGN>(k, t).  The buffers
// are free on entry and hold intermediate passes on exit.  Every thread of
// the block must call this (block-wide barriers).
template <int LGN, bool INV, int NA, int LGNS = 0>
__device__ __forceinline__ void transform(float2 (&v)[NA][E], float2 *const (&buf)[NA], int t,
                                          const float2 *__restrict__ tw)
{
    using P = Pass<LGN, LGNS>;
#pragma unroll
    for (int a = 0; a < NA; ++a) pass_compute<LGN, LGNS, INV>(v[a], t, tw);
    if constexpr (!P::LAST) {
        __syncthreads();  // every thread has read the previous contents
        store_pass<LGN, LGNS, NA>(v, buf, t);
        __syncthreads();
        load_pass<LGN, LGNS + P::LGR, NA>(v, buf, t);
        transform<LGN, INV, NA, LGNS + P::LGR>(v, buf, t, tw + P::TWLEN);
    }
}

// radix (log2) of the last pass of a length-2^lgn transform
__host__ __device__ constexpr int last_lgr(int lgn) { return (lgn & 3) ? (lgn & 3) : 4; }

// element index of register k after transform<LGN>: t + (k / R) n/16 +
// (k mod R) n/R, R the last pass's radix
template <int LGN>
__device__ __forceinline__ int result_index(int k, int t)
{
    constexpr int LGR = last_lgr(LGN);
    return t + (k >> LGR) * (1 << (LGN - 4)) + (k & ((1 << LGR) - 1)) * (1 << (LGN - LGR));
}

// ---- radix-2 stages over four registers, shared by the transforms with four
// elements per thread (here and in pic_spectral_small.cu)
__device__ __forceinline__ constexpr int rev2(int i) { return ((i & 1) << 1) | (i >> 1); }

// a (c -+ i s), - forward, + inverse: w16 for an angle that depends on the
// thread (exact where w16 only swaps or keeps)
template <bool INV>
__device__ __forceinline__ float2 rot(float2 a, float c, float s)
{
    if (!INV) s = -s;
    return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c));
}

// one stage of a radix-2 decimation in frequency over the pairs (v0, v2), (v1, v3)
template <bool INV>
__device__ __forceinline__ void far_pairs(float2 (&v)[4], float c0, float s0, float c1, float s1)
{
    const float2 a = v[0], b = v[1], c = v[2], d = v[3];
    v[0] = cadd(a, c);
    v[1] = cadd(b, d);
    v[2] = rot<INV>(csub(a, c), c0, s0);
    v[3] = rot<INV>(csub(b, d), c1, s1);
}
// and over (v0, v1), (v2, v3)
template <bool INV>
__device__ __forceinline__ void near_pairs(float2 (&v)[4], float c0, float s0)
{
    const float2 a = v[0], b = v[1], c = v[2], d = v[3];
    v[0] = cadd(a, b);
    v[2] = cadd(c, d);
    v[1] = rot<INV>(csub(a, b), c0, s0);
    v[3] = rot<INV>(csub(c, d), c0, s0);
}

// A transform of length 2^LGN as the kernels hold it: n/EL threads with EL
// elements each.  v[a][k] is element in(k, t) before and out(k, t) after run();
// slot(i) is element i's place in a shared buffer of `room` slots.
template <int LGN, int EL>
struct Line;

template <int LGN>
struct Line<LGN, 16> {
    static constexpr int TP = 1 << (LGN - 4);
    static __device__ __forceinline__ int in(int k, int t) { return t + k * TP; }
    static __device__ __forceinline__ int out(int k, int t) { return result_index<LGN>(k, t); }
    static __device__ __forceinline__ int slot(int i) { return pad(i); }
    template <bool INV, int NA>
    static __device__ __forceinline__ void run(float2 (&v)[NA][16], float2 *const (&buf)[NA], int t,
                                               const float2 *__restrict__ tw)
    {
        transform<LGN, INV, NA>(v, buf, t, tw);
    }
};

// Four elements per thread (2^LGN >= 128, whole warps): the passes of
// transform<LGN> in the same order of operations, each radix-16 butterfly
// over four neighbouring lanes and a radix-8 one over two, so that every
// result keeps its bits.  A quarter of the chain per thread and four times
// the threads: for grids that do not fill the GPU.
template <int LGN>
struct Line<LGN, 4> {
    static_assert(LGN >= 7, "whole warps");
    static constexpr int N = 1 << LGN, TP = N / 4;
    static __host__ __device__ constexpr int lgr(int lgns) { return pass_lgr(LGN, lgns); }
    // register k's butterfly and its input and output there, pass lgns
    static __device__ __forceinline__ int fly(int lgns, int k, int t)
    {
        return lgr(lgns) == 4 ? t >> 2 : lgr(lgns) == 3 ? t >> 1 : lgr(lgns) == 2 ? t : t + (k & 1) * TP;
    }
    static __device__ __forceinline__ int rin(int lgns, int k, int t)
    {
        return lgr(lgns) == 4 ? (t & 3) + 4 * k : lgr(lgns) == 3 ? (t & 1) + 2 * k : lgr(lgns) == 2 ? k : k >> 1;
    }
    static __device__ __forceinline__ int rout(int lgns, int k, int t)
    {
        return lgr(lgns) == 4 ? 4 * rev2(k) + rev2(t & 3) : lgr(lgns) == 3 ? 4 * (t & 1) + rev2(k)
             : lgr(lgns) == 2 ? k : k >> 1;
    }
    static __device__ __forceinline__ int src(int lgns, int k, int t)
    {
        return fly(lgns, k, t) + rin(lgns, k, t) * (N >> lgr(lgns));
    }
    static __device__ __forceinline__ int dst(int lgns, int k, int t)
    {
        const int j = fly(lgns, k, t);
        return ((j >> lgns) << (lgns + lgr(lgns))) + (j & ((1 << lgns) - 1)) + (rout(lgns, k, t) << lgns);
    }
    static __host__ __device__ constexpr int last_lgns() { return (LGN - 1) / 4 * 4; }
    static __device__ __forceinline__ int in(int k, int t) { return src(0, k, t); }
    static __device__ __forceinline__ int out(int k, int t) { return dst(last_lgns(), k, t); }
    // four slots between rows of sixteen: the butterflies' lanes on different banks
    static __device__ __forceinline__ int slot(int i) { return i + 4 * (i >> 4); }

    // register q of lane g and register g of lane q change places (four lanes)
    static __device__ __forceinline__ void turn(float2 (&v)[4], int t)
    {
#pragma unroll
        for (int m = 1; m <= 2; m <<= 1)
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int lo = m == 1 ? 2 * p : p, hi = lo + m;
                const bool up = t & m;
                float2 z = up ? v[lo] : v[hi];
                z.x = __shfl_xor_sync(0xffffffffu, z.x, m);
                z.y = __shfl_xor_sync(0xffffffffu, z.y, m);
                if (up)
                    v[lo] = z;
                else
                    v[hi] = z;
            }
    }

    template <bool INV, int NA, int LGNS = 0>
    static __device__ __forceinline__ void run(float2 (&v)[NA][4], float2 *const (&buf)[NA], int t,
                                               const float2 *__restrict__ tw)
    {
        constexpr float C = 0.92387953251128675613f;  // cos(pi / 8)
        constexpr float S = 0.38268343236508977173f;  // sin(pi / 8)
        constexpr float H = 0.70710678118654752440f;  // sqrt(1 / 2)
        constexpr int LGR = lgr(LGNS), NS = 1 << LGNS;
        constexpr bool LAST = LGNS + LGR == LGN;
        if (LGNS > 0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (LGR <= 2 && rin(LGNS, k, 0) == 0) continue;
                float2 w = __ldg(tw + rin(LGNS, k, t) * NS + (fly(LGNS, k, t) & (NS - 1)));
                if (INV) w.y = -w.y;
#pragma unroll
                for (int a = 0; a < NA; ++a) v[a][k] = cmul(v[a][k], w);
            }
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            if (LGR == 4) {
                // stages h = 8 and 4 over inputs q, q + 4, q + 8, q + 12, then
                // h = 2 and 1 over positions 4 q .. 4 q + 3
                const int q = t & 3;
                const float c1 = q == 0 ? 1.f : q == 1 ? C : q == 2 ? H : S;
                const float s1 = q == 0 ? 0.f : q == 1 ? S : q == 2 ? H : C;
                const float c2 = q == 0 ? 1.f : q == 1 ? H : q == 2 ? 0.f : -H;
                const float s2 = q == 0 ? 0.f : q == 2 ? 1.f : H;
                far_pairs<INV>(v[a], c1, s1, -s1, c1);
                near_pairs<INV>(v[a], c2, s2);
                turn(v[a], t);
                far_pairs<INV>(v[a], 1.f, 0.f, 0.f, 1.f);
                near_pairs<INV>(v[a], 1.f, 0.f);
            } else if (LGR == 3) {
                // h = 4 and 2 over inputs q, q + 2, q + 4, q + 6, then h = 1
                // with the other lane
                const bool q = t & 1;
                far_pairs<INV>(v[a], q ? H : 1.f, q ? H : 0.f, q ? -H : 0.f, q ? H : 1.f);
                near_pairs<INV>(v[a], q ? 0.f : 1.f, q ? 1.f : 0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 z = make_float2(__shfl_xor_sync(0xffffffffu, v[a][k].x, 1),
                                                 __shfl_xor_sync(0xffffffffu, v[a][k].y, 1));
                    v[a][k] = q ? csub(z, v[a][k]) : cadd(v[a][k], z);
                }
            } else if (LGR == 2) {
                dft<4, INV>(v[a]);
            } else {
                far_pairs<INV>(v[a], 1.f, 0.f, 1.f, 0.f);
            }
        }
        if constexpr (!LAST) {
            __syncthreads();  // every thread has read the previous contents
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int k = 0; k < 4; ++k) buf[a][slot(dst(LGNS, k, t))] = v[a][k];
            __syncthreads();
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int k = 0; k < 4; ++k) v[a][k] = buf[a][slot(src(LGNS + LGR, k, t))];
            run<INV, NA, LGNS + LGR>(v, buf, t, tw + (LGNS > 0 ? NS << LGR : 0));
        }
    }
};

}  // namespace fft
}  // namespace pic
