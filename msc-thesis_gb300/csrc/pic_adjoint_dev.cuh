// pic_adjoint_dev.cuh -- device functions of the adjoint of the step (CIC
// weights and their gradients, the transposed spectral solve per mode),
// shared by the single-run adjoint (pic_adjoint.cu) and the ensemble adjoint
// (pic_ensemble_adjoint.cu).
#pragma once
#include <cuda_runtime.h>

#include "pic_push_dev.cuh"

namespace pic {

struct Cic {
    int i00, i10, i01, i11;
    float fx, fy;
    bool ok;
};

__device__ __forceinline__ Cic cic_of(int c, float ox, float oy, int nx, int ny)
{
    Cic w;
    const int cx = c & 0xFFFF, cy = c >> 16;
    w.ok = c >= 0 && cx < nx && cy < ny;
    const int cx1 = (cx + 1 == nx) ? 0 : cx + 1, cy1 = (cy + 1 == ny) ? 0 : cy + 1;
    w.i00 = cy * nx + cx;
    w.i10 = cy * nx + cx1;
    w.i01 = cy1 * nx + cx;
    w.i11 = cy1 * nx + cx1;
    w.fx = ox;
    w.fy = oy;
    return w;
}

// sum_k grad w_k s_k, physical units
__device__ __forceinline__ float2 grad_dot(const Cic &w, float s00, float s10, float s01,
                                           float s11, float inv_dx, float inv_dy)
{
    const float fx = w.fx, fy = w.fy;
    return make_float2(((1.f - fy) * (s10 - s00) + fy * (s11 - s01)) * inv_dx,
                       ((1.f - fx) * (s01 - s00) + fx * (s11 - s10)) * inv_dy);
}

// One mode of psi = S^T g, the transpose of the field solve E = S rho:
// psi^ = i (kx g^x + ky g^y) / (eps0 N k^2) with the Nyquist derivative
// zeroed as in the forward solve and the zero mode removed (N folded in).
__device__ __forceinline__ float2 adj_mode(float2 a, float2 b, int mx, int my, int nx, int ny,
                                           float kx1, float ky1, float inv_eps0_n, bool zero_mode)
{
    const bool nx_even = (nx & 1) == 0, ny_even = (ny & 1) == 0;
    const int sy = (2 * my <= ny) ? my : my - ny;
    const float kx = kx1 * (float)mx, ky = ky1 * (float)sy;
    const float kxe = (nx_even && 2 * mx == nx) ? 0.f : kx;
    const float kye = (ny_even && 2 * my == ny) ? 0.f : ky;
    const float hr = kxe * a.x + kye * b.x, hi = kxe * a.y + kye * b.y;
    const float inv = zero_mode ? 0.f : inv_eps0_n / (kx * kx + ky * ky);
    return make_float2(-hi * inv, hr * inv);  // i (hr + i hi)
}

// ---- the kick's transpose, one block of a push grid
struct KickArgs {
    const int32_t *cell;
    const float *ox, *oy;
    float *vx, *vy;              // un-kicked in place by the reversal (UNKICK)
    float *ax, *ay, *avx, *avy;  // adjoint state
};
struct KickGeo {
    PushGeo G;        // grid, field and window (no density, no step coefficients)
    float *gx, *gy;   // scatter planes
    float qm_dt;      // dt q/m of the reversed kick
    float muc, ddt;   // mu = muc a_v; drift adjoint a_v += ddt a_x
    float inv_dx, inv_dy;
};

// Shared memory of a kick block: E at the window's nodes, then five words per
// node, of which four are used (an odd stride: neighbouring nodes on
// different banks): the high and low halves of the fixed-point sums of the
// node's x and y scatter.
__host__ __device__ __forceinline__ size_t kick_bytes(int wcx, int wcy)
{
    return (size_t)(wcx + 1) * (wcy + 1) * (sizeof(float2) + 5 * sizeof(unsigned)) + 16;
}

// adds v (|v| < 2^31 / scale) to the split fixed-point sum at m
__device__ __forceinline__ void add_fixed(unsigned *m, float v, float scale)
{
    const int q = __float2int_rn(v * scale);
    atomicAdd(m, (unsigned)(q >> 16));
    atomicAdd(m + 1, (unsigned)q & 0xFFFFu);
}

__device__ __forceinline__ float fixed_sum(const unsigned *m, float inv_scale)
{
    return (float)(((long long)(int)m[0] << 16) + (long long)m[1]) * inv_scale;
}

// Drift adjoint, kick transpose (scatter of mu and local term) and, with
// UNKICK, the reversal of the kick, of particles [base, end) (multiples of 4
// from base).  E comes from the block's window, and the scatter is summed
// there in fixed point: shared-memory integer adds are native, float ones are
// compare-and-swap loops.  A first pass over the block's adjoint velocities
// finds their largest magnitude, which sets the scale (31 bits for the largest
// mu, at most 32768 particles a block: the 16-bit halves cannot overflow); it
// also brings the four arrays into L2 for the second.  A contribution is rounded
// to 2^-31 of the largest at most, and the sums are exact from there and
// independent of order.  So that a few values far above the others do not
// take their bits, the largest counts as no more than 2^KICK_SPAN times the
// geometric mean (by the mean exponent of the nonzero values; it is 2^2 to 2^5
// times that in ordinary runs): the rounding is then below 2^-24 of that mean, as
// a float's is of values of its size.  Particles above that, blocks whose largest value is not finite or too small
// to scale, and particles outside the window add to the grid in float.  8 runs
// of up to 256^2 x 64 (10.3 M particles): 171 us against 316 us with float sums
// over a warp's equal cells first and compare-and-swap adds of the rest (60
// bytes per particle: 91 us).
constexpr int KICK_SPAN = 6;

template <bool UNKICK>
__device__ __forceinline__ void adj_kick_block(const KickArgs &A, const KickGeo &K,
                                               unsigned char *smem, long long base, long long end,
                                               int anc)
{
    __shared__ unsigned s_max, s_exp, s_cnt;
    const PushGeo &G = K.G;
    const Window W = setup_window(G, smem, anc);
    if (threadIdx.x == 0) s_max = s_exp = s_cnt = 0u;
    load_window<true, false>(G, W);
    if (W.on)
        for (int i = threadIdx.x; i < 5 * W.nw; i += blockDim.x) W.sM[i] = 0u;
    __syncthreads();
    // largest |a_v| after the drift, as its bits (a NaN above all); sum of the
    // biased exponents and number of the normal values
    unsigned big = 0u, exps = 0u, cnt = 0u;
    for (long long q = base + 4ll * threadIdx.x; q < end; q += 4ll * blockDim.x) {
        const float4 x4 = *reinterpret_cast<const float4 *>(A.ax + q);
        const float4 y4 = *reinterpret_cast<const float4 *>(A.ay + q);
        const float4 u4 = *reinterpret_cast<const float4 *>(A.avx + q);
        const float4 w4 = *reinterpret_cast<const float4 *>(A.avy + q);
        const float m[8] = {fmaf(K.ddt, x4.x, u4.x), fmaf(K.ddt, x4.y, u4.y), fmaf(K.ddt, x4.z, u4.z),
                            fmaf(K.ddt, x4.w, u4.w), fmaf(K.ddt, y4.x, w4.x), fmaf(K.ddt, y4.y, w4.y),
                            fmaf(K.ddt, y4.z, w4.z), fmaf(K.ddt, y4.w, w4.w)};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned bits = __float_as_uint(m[k]) & 0x7FFFFFFFu, ex = bits >> 23;
            big = max(big, bits);
            exps += ex;
            cnt += min(ex, 1u);
        }
    }
    big = __reduce_max_sync(0xffffffffu, big);
    exps = __reduce_add_sync(0xffffffffu, exps);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_max, big);
        atomicAdd(&s_exp, exps);
        atomicAdd(&s_cnt, cnt);
    }
    __syncthreads();
    // the values summed in fixed point are below 2^e, e in [-94, 128]; scale = 2^(31 - e)
    big = s_max;
    if (s_cnt && big < 0x7F800000u) big = min(big, min(s_exp / s_cnt + KICK_SPAN + 1, 254u) << 23);
    const float top = __uint_as_float(big) * fabsf(K.muc);
    const int e = (int)(__float_as_uint(top) >> 23) - 126;
    const bool fixed = W.on && e >= -94 && e <= 128;
    const float scale = __uint_as_float((unsigned)(158 - e) << 23);
    const float inv_scale = __uint_as_float((unsigned)(96 + e) << 23);
    const float below = __uint_as_float((unsigned)(127 + e) << 23);  // 2^e
    const int nx = G.nx, ny = G.ny;
    for (long long q = base + 4ll * threadIdx.x; q < end; q += 4ll * blockDim.x) {
        const int4 c4 = *reinterpret_cast<const int4 *>(A.cell + q);
        const float4 a4 = *reinterpret_cast<const float4 *>(A.ox + q);
        const float4 b4 = *reinterpret_cast<const float4 *>(A.oy + q);
        const float4 x4 = *reinterpret_cast<const float4 *>(A.ax + q);
        const float4 y4 = *reinterpret_cast<const float4 *>(A.ay + q);
        const float4 u4 = *reinterpret_cast<const float4 *>(A.avx + q);
        const float4 w4 = *reinterpret_cast<const float4 *>(A.avy + q);
        float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f), r4 = p4;
        if (UNKICK) {
            p4 = *reinterpret_cast<const float4 *>(A.vx + q);
            r4 = *reinterpret_cast<const float4 *>(A.vy + q);
        }
        const int cc[4] = {c4.x, c4.y, c4.z, c4.w};
        const float ox[4] = {a4.x, a4.y, a4.z, a4.w}, oy[4] = {b4.x, b4.y, b4.z, b4.w};
        float ax[4] = {x4.x, x4.y, x4.z, x4.w}, ay[4] = {y4.x, y4.y, y4.z, y4.w};
        float avx[4] = {u4.x, u4.y, u4.z, u4.w}, avy[4] = {w4.x, w4.y, w4.z, w4.w};
        float vx[4] = {p4.x, p4.y, p4.z, p4.w}, vy[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = cc[j];
            const int cx = c & 0xFFFF, cy = c >> 16;
            if (c < 0 || cx >= nx || cy >= ny) continue;
            const float avxj = fmaf(K.ddt, ax[j], avx[j]), avyj = fmaf(K.ddt, ay[j], avy[j]);
            const float mx = K.muc * avxj, my = K.muc * avyj;
            const float gx = 1.f - ox[j], gy = 1.f - oy[j];
            const float w00 = gx * gy, w10 = ox[j] * gy, w01 = gx * oy[j], w11 = ox[j] * oy[j];
            float2 e00, e10, e01, e11;
            int dxl, dyl;
            window_coords(G, W, cx, cy, dxl, dyl);
            const bool in = (unsigned)dxl < W.wcx && (unsigned)dyl < W.wcy;
            const int l = in ? dyl * W.nwx + dxl : 0;
            const Cic w = cic_of(c, 0.f, 0.f, nx, ny);
            if (in) {
                e00 = W.sE[l];
                e10 = W.sE[l + 1];
                e01 = W.sE[l + W.nwx];
                e11 = W.sE[l + W.nwx + 1];
            } else {
                e00 = make_float2(G.ex[w.i00], G.ey[w.i00]);
                e10 = make_float2(G.ex[w.i10], G.ey[w.i10]);
                e01 = make_float2(G.ex[w.i01], G.ey[w.i01]);
                e11 = make_float2(G.ex[w.i11], G.ey[w.i11]);
            }
            if (in && fixed && fmaxf(fabsf(mx), fabsf(my)) < below) {
                unsigned *m0 = W.sM + 5 * l, *m1 = m0 + 5 * W.nwx;
                add_fixed(m0, w00 * mx, scale);
                add_fixed(m0 + 2, w00 * my, scale);
                add_fixed(m0 + 5, w10 * mx, scale);
                add_fixed(m0 + 7, w10 * my, scale);
                add_fixed(m1, w01 * mx, scale);
                add_fixed(m1 + 2, w01 * my, scale);
                add_fixed(m1 + 5, w11 * mx, scale);
                add_fixed(m1 + 7, w11 * my, scale);
            } else {
                atomicAdd(K.gx + w.i00, w00 * mx);
                atomicAdd(K.gy + w.i00, w00 * my);
                atomicAdd(K.gx + w.i10, w10 * mx);
                atomicAdd(K.gy + w.i10, w10 * my);
                atomicAdd(K.gx + w.i01, w01 * mx);
                atomicAdd(K.gy + w.i01, w01 * my);
                atomicAdd(K.gx + w.i11, w11 * mx);
                atomicAdd(K.gy + w.i11, w11 * my);
            }
            const float s00 = e00.x * mx + e00.y * my, s10 = e10.x * mx + e10.y * my;
            const float s01 = e01.x * mx + e01.y * my, s11 = e11.x * mx + e11.y * my;
            ax[j] += (gy * (s10 - s00) + oy[j] * (s11 - s01)) * K.inv_dx;
            ay[j] += (gx * (s01 - s00) + ox[j] * (s11 - s10)) * K.inv_dy;
            avx[j] = avxj;
            avy[j] = avyj;
            if (UNKICK) {  // the push's gather, then the kick taken back
                const float Ex = gy * fmaf(gx, e00.x, ox[j] * e10.x) + oy[j] * fmaf(gx, e01.x, ox[j] * e11.x);
                const float Ey = gy * fmaf(gx, e00.y, ox[j] * e10.y) + oy[j] * fmaf(gx, e01.y, ox[j] * e11.y);
                vx[j] = fmaf(-K.qm_dt, Ex, vx[j]);
                vy[j] = fmaf(-K.qm_dt, Ey, vy[j]);
            }
        }
        *reinterpret_cast<float4 *>(A.ax + q) = make_float4(ax[0], ax[1], ax[2], ax[3]);
        *reinterpret_cast<float4 *>(A.ay + q) = make_float4(ay[0], ay[1], ay[2], ay[3]);
        *reinterpret_cast<float4 *>(A.avx + q) = make_float4(avx[0], avx[1], avx[2], avx[3]);
        *reinterpret_cast<float4 *>(A.avy + q) = make_float4(avy[0], avy[1], avy[2], avy[3]);
        if (UNKICK) {
            *reinterpret_cast<float4 *>(A.vx + q) = make_float4(vx[0], vx[1], vx[2], vx[3]);
            *reinterpret_cast<float4 *>(A.vy + q) = make_float4(vy[0], vy[1], vy[2], vy[3]);
        }
    }
    if (!fixed) return;
    __syncthreads();
    WindowWalk w(W);
    for (int i = threadIdx.x; i < W.nw; i += blockDim.x, w.next(W)) {
        const float fx = fixed_sum(W.sM + 5 * i, inv_scale), fy = fixed_sum(W.sM + 5 * i + 2, inv_scale);
        if (fx == 0.f && fy == 0.f) continue;
        const size_t o = w.node(W, nx, ny);
        if (fx != 0.f) atomicAdd(K.gx + o, fx);
        if (fy != 0.f) atomicAdd(K.gy + o, fy);
    }
}

}  // namespace pic
