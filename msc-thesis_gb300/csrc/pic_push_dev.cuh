// pic_push_dev.cuh -- device functions of the fused gather + push + deposit
// pass, shared by the single-run kernels (pic_push.cu) and the ensemble
// kernels (pic_ensemble.cu).  The arithmetic and the work decomposition are
// described at the top of pic_push.cu.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "pic_internal.cuh"

namespace pic {

struct Cic4 {
    unsigned long long w00, w10, w01, w11;
};

// Node weights of `cnt` particles in one cell from their sums of fx, fy, fx*fy.
__device__ __forceinline__ Cic4 cic_weights(unsigned cnt, unsigned sfx, unsigned sfy,
                                            unsigned long long sxy)
{
    Cic4 W;
    W.w11 = sxy;
    W.w10 = ((unsigned long long)sfx << 16) - sxy;
    W.w01 = ((unsigned long long)sfy << 16) - sxy;
    W.w00 = ((unsigned long long)cnt << 32) - ((unsigned long long)(sfx + sfy) << 16) + sxy;
    return W;
}

// rint(o 2^16) for an in-cell offset o in [0, 1), round to nearest even:
// adding 1.5 2^23 in the same fused operation leaves the rounded integer in
// the low mantissa bits (one rounding of the exact o 2^16 + 1.5 2^23, whose
// unit in the last place is 1), the same value as __float2uint_rn(o * 65536)
__device__ __forceinline__ unsigned offset_fixed(float o)
{
    return __float_as_uint(fmaf(o, 65536.0f, 12582912.0f)) - 0x4B400000u;
}

__device__ __forceinline__ void deposit_global(unsigned long long *rho, int nx, int ny, int cx,
                                               int cy, const Cic4 &W, unsigned long long q)
{
    const int cx1 = (cx + 1 == nx) ? 0 : cx + 1;
    const int cy1 = (cy + 1 == ny) ? 0 : cy + 1;
    atomicAdd(rho + (size_t)cy * nx + cx, W.w00 * q);
    atomicAdd(rho + (size_t)cy * nx + cx1, W.w10 * q);
    atomicAdd(rho + (size_t)cy1 * nx + cx, W.w01 * q);
    atomicAdd(rho + (size_t)cy1 * nx + cx1, W.w11 * q);
}

// Per-run part of a push pass: the grid, its field and density, the
// diagnostics, the tile window and the step coefficients.
struct PushGeo {
    const float *ex, *ey;
    unsigned long long *rho;
    DevState *dev;
    int nx, ny, tw, th, hx, hy, wcx, wcy;  // window halo hx, hy; size wcx x wcy cells
    float qm_dt, dtdx, dtdy;
    unsigned long long qmul;  // q_int as two's complement
    double ke_scale, p_scale; // m/4, m/2 (0 disables the diagnostics)
    uint32_t *recount;        // per cell key: counts kept current across cell changes (or null)
    int ntx;                  // tiles along x (cell keys of recount)
};

// tile-major cell key (the sort's key; divisions, for the rare cell changes)
__device__ __forceinline__ int push_cell_key(int cx, int cy, const PushGeo &A)
{
    const int tx = cx / A.tw, ty = cy / A.th;
    return ((ty * A.ntx + tx) * A.th + (cy - ty * A.th)) * A.tw + (cx - tx * A.tw);
}

// Particle arrays of a push pass (and, for a single run, its PushGeo).
struct PushArgs {
    const int32_t *cin;
    const float *oxin, *oyin, *vxin, *vyin;
    int32_t *cout;
    float *oxout, *oyout, *vxout, *vyout;
    const uint32_t *pidin;  // copied to pidout when non-null (out-of-place pass)
    uint32_t *pidout;
    const float *vzin;      // copied to vzout when non-null
    float *vzout;
    const int32_t *anchor;
    const long long *d_n;
    int chunk;
    PushGeo geo;
};

// Shared-memory window of a push block (layout: window_bytes), anchored at
// the tile of the block's first particle.  The deposit keeps per-cell CIC
// moments in sM, five words per cell: one address for a particle's five
// atomics (the rest is immediate offsets), and the odd stride puts
// neighbouring cells on different banks (the adjoint's kick keeps its sums
// there, see kick_bytes).  wcx is 0 where the block has no window (!on), so that
// no cell lies in it.
struct Window {
    float2 *sE;
    unsigned *sM;
    int wx0, wy0, nwx, nw, nc;
    unsigned wcx, wcy;
    bool on;
};

__device__ __forceinline__ Window setup_window(const PushGeo &A, unsigned char *smem, int anc)
{
    Window W;
    W.nwx = A.wcx + 1;
    W.nw = W.nwx * (A.wcy + 1);
    W.sE = reinterpret_cast<float2 *>(smem);
    W.sM = reinterpret_cast<unsigned *>(smem + (size_t)W.nw * sizeof(float2));
    W.nc = A.wcx * A.wcy;
    W.on = anc >= 0;
    W.wcx = W.on ? A.wcx : 0;
    W.wcy = A.wcy;
    W.wx0 = W.wy0 = 0;
    if (W.on) {
        int wx0 = (anc & 0xFFFF) * A.tw - A.hx, wy0 = (anc >> 16) * A.th - A.hy;
        wx0 %= A.nx;
        if (wx0 < 0) wx0 += A.nx;
        wy0 %= A.ny;
        if (wy0 < 0) wy0 += A.ny;
        W.wx0 = wx0;
        W.wy0 = wy0;
    }
    return W;
}

// A value that an earlier kernel of the chain wrote: a late kernel (see
// pdl_wait) reads it from L2.
template <bool LATE, class T>
__device__ __forceinline__ T ld(const T *p)
{
    return LATE ? __ldcg(p) : *p;
}

// Walks the window's nodes i = threadIdx.x, threadIdx.x + blockDim.x, ...
// with their grid node (gx, gy), advanced incrementally (the divisions run
// once per thread, not once per node).
struct WindowWalk {
    int a, b, da, db;  // window column and row, and their step
    __device__ __forceinline__ WindowWalk(const Window &W)
    {
        db = blockDim.x / W.nwx;
        da = blockDim.x - db * W.nwx;
        b = threadIdx.x / W.nwx;
        a = threadIdx.x - b * W.nwx;
    }
    __device__ __forceinline__ void next(const Window &W)
    {
        a += da;
        b += db;
        if (a >= W.nwx) {
            a -= W.nwx;
            ++b;
        }
    }
    // grid node of the current window node (wx0 < nx, wy0 < ny)
    __device__ __forceinline__ size_t node(const Window &W, int nx, int ny) const
    {
        int gx = W.wx0 + a, gy = W.wy0 + b;
        while (gx >= nx) gx -= nx;
        while (gy >= ny) gy -= ny;
        return (size_t)gy * nx + gx;
    }
};

template <bool GATHER, bool DEPOSIT, bool LATE = false>
__device__ __forceinline__ void load_window(const PushGeo &A, const Window &W)
{
    if (!W.on) return;
    if (GATHER) {
        WindowWalk w(W);
        for (int i = threadIdx.x; i < W.nw; i += blockDim.x, w.next(W)) {
            const size_t g = w.node(W, A.nx, A.ny);
            W.sE[i] = make_float2(ld<LATE>(A.ex + g), ld<LATE>(A.ey + g));
        }
    }
    if (DEPOSIT) {  // 8-byte stores (the moments start on 8 bytes)
        const int words = 5 * W.nc;
        for (int i = threadIdx.x; 2 * i + 1 < words; i += blockDim.x)
            reinterpret_cast<uint2 *>(W.sM)[i] = make_uint2(0u, 0u);
        if ((words & 1) && threadIdx.x == 0) W.sM[words - 1] = 0u;
    }
}

// Window coordinates of cell (cx, cy): its column and row counted from the
// window's first (periodically), so that it lies in the window exactly
// when 0 <= dxl < wcx and 0 <= dyl < wcy.
__device__ __forceinline__ void window_coords(const PushGeo &A, const Window &W, int cx, int cy,
                                              int &dxl, int &dyl)
{
    dxl = cx - W.wx0;
    dyl = cy - W.wy0;
    if (dxl < 0) dxl += A.nx;
    if (dyl < 0) dyl += A.ny;
}

// five shared atomics: a group's moments into its cell of the window
__device__ __forceinline__ void add_moments(unsigned *m, unsigned cnt, unsigned sfx, unsigned sfy,
                                            unsigned long long sxy)
{
    atomicAdd(m, cnt);
    atomicAdd(m + 1, sfx);
    atomicAdd(m + 2, sfy);
    atomicAdd(m + 3, (unsigned)(sxy & 0xFFFFull));
    atomicAdd(m + 4, (unsigned)(sxy >> 16));
}

// One group of `cnt` particles in cell (cx, cy), window coordinates (dxl,
// dyl), with sums fx, fy, fx*fy: its moments added to the window's cell
// (five shared atomics; the node weights are linear in them and are formed
// at the flush), or its node weights straight to the grid outside the
// window.  The window coordinates may run one carry past the range of
// window_coords (a column or row from -1 to nx): any value maps to the
// grid node the flush gives it, and values outside [0, wcx) x [0, wcy)
// take the grid path.
__device__ __forceinline__ void deposit_group(const PushGeo &A, const Window &W, int cx, int cy,
                                              int dxl, int dyl, unsigned cnt, unsigned sfx,
                                              unsigned sfy, unsigned long long sxy)
{
    if ((unsigned)dxl < W.wcx && (unsigned)dyl < W.wcy) {
        add_moments(W.sM + 5 * (dyl * A.wcx + dxl), cnt, sfx, sfy, sxy);
    } else {
        deposit_global(A.rho, A.nx, A.ny, cx, cy, cic_weights(cnt, sfx, sfy, sxy), A.qmul);
    }
}

// Sum of the lanes' (count, sum fx, sum fy, sum fx*fy) over each maximal run
// of consecutive lanes with the same key; returns true on the run's first
// lane, which holds the run's total.  All 32 lanes must call it (full-warp
// shuffles and ballot); key -1 marks a lane without a group.  Runs are
// exact for any key sequence: lane i adds the partial of lane i + o only
// while i + o lies before the next run start, so no lane is counted twice.
__device__ __forceinline__ bool warp_group_sum(int key, unsigned &c, unsigned &fx, unsigned &fy,
                                               unsigned long long &xy)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(full, key, 1);
    const bool head = lane == 0 || key != prev;
    const unsigned heads = __ballot_sync(full, head);
    const unsigned after = heads & (0xfffffffeu << lane);  // run starts after this lane
    const int seg_end = after ? __ffs(after) - 1 : 32;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned c2 = __shfl_down_sync(full, c, o);
        const unsigned fx2 = __shfl_down_sync(full, fx, o);
        const unsigned fy2 = __shfl_down_sync(full, fy, o);
        const unsigned long long xy2 = __shfl_down_sync(full, xy, o);
        if (lane + o < seg_end) {
            c += c2;
            fx += fx2;
            fy += fy2;
            xy += xy2;
        }
    }
    return head;
}

// v mod n for a cell coordinate that left [0, n) (0 <= result < n): two
// float quotients, each off by a few units at most, then one correction.
__device__ __forceinline__ int wrap_cell(int v, int n)
{
    const float inv = __fdividef(1.0f, (float)n);
#pragma unroll
    for (int k = 0; k < 2; ++k)
        v -= (int)((unsigned)n * (unsigned)(int)floorf((float)v * inv));
    if (v < 0) v += n;
    if (v >= n) v -= n;
    return v;
}

// One particle with its cell on the grid: gather, push, and its new cell,
// window coordinates and fixed-point offsets to `deposit`.  One branch for
// all that a drift makes rare (an offset rounded up to 1, a cell across the
// boundary).
template <bool GATHER, bool DEPOSIT, bool MOVE, bool LATE, class F>
__device__ __forceinline__ void push_one(const PushGeo &A, const Window &W, int &cell, float &x,
                                         float &y, float &u, float &v, float &ke, float &px,
                                         float &py, F &&deposit)
{
    const int nx = A.nx, ny = A.ny;
    const int c = cell;
    int cx = c & 0xFFFF, cy = c >> 16;
    float ox = x, oy = y, vx = u, vy = v;
    int dxl, dyl;  // window coordinates, advanced with the cell below
    window_coords(A, W, cx, cy, dxl, dyl);
    if (MOVE && GATHER) {
        const float gx = 1.f - ox, gy = 1.f - oy;
        float2 e00, e10, e01, e11;
        if ((unsigned)dxl < W.wcx && (unsigned)dyl < W.wcy) {
            const float2 *e = W.sE + dyl * W.nwx + dxl;
            e00 = e[0];
            e10 = e[1];
            e01 = e[W.nwx];
            e11 = e[W.nwx + 1];
        } else {
            const int cx1 = (cx + 1 == nx) ? 0 : cx + 1;
            const int cy1 = (cy + 1 == ny) ? 0 : cy + 1;
            const int i00 = cy * nx + cx, i10 = cy * nx + cx1;
            const int i01 = cy1 * nx + cx, i11 = cy1 * nx + cx1;
            e00 = make_float2(ld<LATE>(A.ex + i00), ld<LATE>(A.ey + i00));
            e10 = make_float2(ld<LATE>(A.ex + i10), ld<LATE>(A.ey + i10));
            e01 = make_float2(ld<LATE>(A.ex + i01), ld<LATE>(A.ey + i01));
            e11 = make_float2(ld<LATE>(A.ex + i11), ld<LATE>(A.ey + i11));
        }
        const float Ex = gy * fmaf(gx, e00.x, ox * e10.x) + oy * fmaf(gx, e01.x, ox * e11.x);
        const float Ey = gy * fmaf(gx, e00.y, ox * e10.y) + oy * fmaf(gx, e01.y, ox * e11.y);
        const float vx0 = vx, vy0 = vy;
        vx = fmaf(A.qm_dt, Ex, vx);
        vy = fmaf(A.qm_dt, Ey, vy);
        ke = fmaf(vx0, vx0, fmaf(vy0, vy0, fmaf(vx, vx, fmaf(vy, vy, ke))));
        px += vx0 + vx;
        py += vy0 + vy;
    } else if (MOVE) {
        ke = fmaf(2.f * vx, vx, fmaf(2.f * vy, vy, ke));
        px = fmaf(2.f, vx, px);
        py = fmaf(2.f, vy, py);
    }
    if (MOVE) {
        // drift in cell units; carry whole cells into the index (a
        // non-finite velocity shows in the thread's kinetic-energy sum)
        ox = fmaf(vx, A.dtdx, ox);
        oy = fmaf(vy, A.dtdy, oy);
        const float sx = floorf(ox), sy = floorf(oy);
        ox -= sx;
        oy -= sy;
        const int kx = (int)sx, ky = (int)sy;
        cx += kx;
        cy += ky;
        dxl += kx;
        dyl += ky;
        if (fmaxf(ox, oy) >= 1.f || (unsigned)cx >= (unsigned)nx || (unsigned)cy >= (unsigned)ny) {
            if (ox >= 1.f) { ox -= 1.f; ++cx; ++dxl; }
            if (oy >= 1.f) { oy -= 1.f; ++cy; ++dyl; }
            if ((unsigned)cx >= (unsigned)nx) cx = wrap_cell(cx, nx);
            if ((unsigned)cy >= (unsigned)ny) cy = wrap_cell(cy, ny);
        }
        const int cn = cx | (cy << 16);
        if (!GATHER && !DEPOSIT && A.recount && cn != c) {  // a neutral that changed cells
            atomicAdd(A.recount + push_cell_key(cx, cy, A), 1u);
            atomicSub(A.recount + push_cell_key(c & 0xFFFF, c >> 16, A), 1u);
        }
        cell = cn;
        x = ox;
        y = oy;
        u = vx;
        v = vy;
    }
    if (DEPOSIT) deposit(cx, cy, dxl, dyl, offset_fixed(ox), offset_fixed(oy));
}

// Four particles with their cells on the grid, each deposited by itself: on
// row-sorted particles a quad rarely shares a cell, and collecting those that
// do in registers first, as push_grouped does, costs divergent code on every
// quad and registers that spill.  2048^2 x 32, sort every 20: 1.094 -> 1.018 ms
// per step (chunk 16384; with the slow slots out of line and one address per
// quad and per deposit); collected per quad as before 1.077, with spills up to
// 1.211.
template <bool GATHER, bool DEPOSIT, bool MOVE, bool LATE>
__device__ __forceinline__ void push_four(const PushGeo &A, const Window &W, int (&cc)[4],
                                          float (&xo)[4], float (&yo)[4], float (&xv)[4],
                                          float (&yv)[4], float &ke, float &px, float &py)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        push_one<GATHER, DEPOSIT, MOVE, LATE>(A, W, cc[j], xo[j], yo[j], xv[j], yv[j], ke, px, py,
                                        [&](int cx, int cy, int dxl, int dyl, unsigned fx, unsigned fy) {
            deposit_group(A, W, cx, cy, dxl, dyl, 1u, fx, fy, (unsigned long long)fx * fy);
        });
}

// Four slots of which some are empty or corrupt (the array's last quad): the
// live ones one at a time through push_one, from local memory, so that the
// code that nearly every quad runs stays small.
template <bool GATHER, bool DEPOSIT, bool MOVE, bool LATE>
__device__ __forceinline__ void push_slots(const PushGeo &A, const Window &W, int (&cc)[4],
                                           float (&xo)[4], float (&yo)[4], float (&xv)[4],
                                           float (&yv)[4], float &ke, float &px, float &py, bool &bad)
{
    int c[4];
    float p[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        c[j] = cc[j];
        p[0][j] = xo[j], p[1][j] = yo[j], p[2][j] = xv[j], p[3][j] = yv[j];
    }
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        if (c[j] < 0) continue;  // empty slot
        if ((c[j] & 0xFFFF) >= A.nx || (c[j] >> 16) >= A.ny) {  // corrupt: flag, leave untouched
            bad = true;
            atomicOr(&A.dev->err, (unsigned)PIC_DEVERR_CELL);
            continue;
        }
        push_one<GATHER, DEPOSIT, MOVE, LATE>(A, W, c[j], p[0][j], p[1][j], p[2][j], p[3][j], ke, px, py,
                                        [&](int cx, int cy, int dxl, int dyl, unsigned fx, unsigned fy) {
            deposit_group(A, W, cx, cy, dxl, dyl, 1u, fx, fy, (unsigned long long)fx * fy);
        });
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        cc[j] = c[j];
        xo[j] = p[0][j], yo[j] = p[1][j], xv[j] = p[2][j], yv[j] = p[3][j];
    }
}

// Four slots, any of them empty or corrupt, for AGG: those that share the first
// one's new cell are collected in registers and these groups summed across
// the warp (warp_group_sum) before the deposit, so that a warp whose particles
// share a cell issues one set of atomics instead of 32 conflicting ones.  Every
// lane of the warp calls it together.
template <bool GATHER>
__device__ __forceinline__ void push_grouped(const PushGeo &A, const Window &W, int (&cc)[4],
                                             float (&xo)[4], float (&yo)[4], float (&xv)[4],
                                             float (&yv)[4], float &ke, float &px, float &py, bool &bad)
{
    unsigned gcnt = 0u, gfx = 0u, gfy = 0u;
    unsigned long long gxy = 0ull;
    int gkey = -1, gdx = 0, gdy = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (cc[j] < 0) continue;  // empty slot
        if ((cc[j] & 0xFFFF) >= A.nx || (cc[j] >> 16) >= A.ny) {  // corrupt: flag, leave untouched
            bad = true;
            atomicOr(&A.dev->err, (unsigned)PIC_DEVERR_CELL);
            continue;
        }
        push_one<GATHER, true, true, false>(A, W, cc[j], xo[j], yo[j], xv[j], yv[j], ke, px, py,
                                            [&](int cx, int cy, int dxl, int dyl, unsigned fx, unsigned fy) {
            const unsigned long long fxy = (unsigned long long)fx * fy;
            const int cn = cx | (cy << 16);
            if (gkey < 0) {
                gkey = cn;
                gdx = dxl;
                gdy = dyl;
            }
            if (cn == gkey) {
                ++gcnt;
                gfx += fx;
                gfy += fy;
                gxy += fxy;
            } else {
                deposit_group(A, W, cx, cy, dxl, dyl, 1u, fx, fy, fxy);
            }
        });
    }
    if (warp_group_sum(gcnt ? gkey : -1, gcnt, gfx, gfy, gxy) && gcnt)
        deposit_group(A, W, gkey & 0xFFFF, gkey >> 16, gdx, gdy, gcnt, gfx, gfy, gxy);
}

// byte offset `o` into one field's array, whose block starts at the uniform
// pointer `p` (one 32-bit offset then serves all of a quad's loads and stores)
template <class T, class P>
__device__ __forceinline__ T &at(P *p, unsigned o)
{
    return *reinterpret_cast<T *>(reinterpret_cast<char *>(const_cast<std::remove_const_t<P> *>(p)) + o);
}

template <bool LATE>
__device__ __forceinline__ void store_quad(const PushArgs &A, long long base, unsigned o,
                                           const int (&cc)[4], const float (&xo)[4],
                                           const float (&yo)[4], const float (&xv)[4],
                                           const float (&yv)[4])
{
    at<int4>(A.cout + base, o) = make_int4(cc[0], cc[1], cc[2], cc[3]);
    at<float4>(A.oxout + base, o) = make_float4(xo[0], xo[1], xo[2], xo[3]);
    at<float4>(A.oyout + base, o) = make_float4(yo[0], yo[1], yo[2], yo[3]);
    at<float4>(A.vxout + base, o) = make_float4(xv[0], xv[1], xv[2], xv[3]);
    at<float4>(A.vyout + base, o) = make_float4(yv[0], yv[1], yv[2], yv[3]);
    if (A.pidin) at<uint4>(A.pidout + base, o) = ld<LATE>(&at<uint4>(A.pidin + base, o));
    if (A.vzin) at<float4>(A.vzout + base, o) = ld<LATE>(&at<float4>(A.vzin + base, o));
}

// end of a block: diagnostics reduction, error flags, window flush
template <bool DEPOSIT>
__device__ __forceinline__ void finish_block(const PushGeo &A, const Window &W, double *sAcc,
                                             float ke, float px, float py, bool bad)
{
    if (A.ke_scale != 0.0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ke += __shfl_xor_sync(0xffffffffu, ke, o);
            px += __shfl_xor_sync(0xffffffffu, px, o);
            py += __shfl_xor_sync(0xffffffffu, py, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(sAcc + 0, (double)ke);
            atomicAdd(sAcc + 1, (double)px);
            atomicAdd(sAcc + 2, (double)py);
        }
    }
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    if (threadIdx.x == 0) {
        if (A.ke_scale != 0.0) {
            const int sl = acc_slot();
            atomicAdd(&A.dev->ke[sl], sAcc[0] * A.ke_scale);
            atomicAdd(&A.dev->px[sl], sAcc[1] * A.p_scale);
            atomicAdd(&A.dev->py[sl], sAcc[2] * A.p_scale);
        }
        if (any_bad) atomicOr(&A.dev->err, (unsigned)PIC_DEVERR_NAN);
    }
    if (DEPOSIT && W.on) {
        // node (a, b) takes w00 of cell (a, b), w10 of (a-1, b), w01 of
        // (a, b-1) and w11 of (a-1, b-1), those inside the window
        const int wcx = A.wcx, wcy = A.wcy;
        const unsigned *m = W.sM;
        auto sxy = [&](int l) { return ((unsigned long long)m[5 * l + 4] << 16) + m[5 * l + 3]; };
        WindowWalk w(W);
        for (int i = threadIdx.x; i < W.nw; i += blockDim.x, w.next(W)) {
            const int a = w.a, b = w.b;
            unsigned long long v = 0ull;
            if (a < wcx && b < wcy) {
                const int l = b * wcx + a;
                v += ((unsigned long long)m[5 * l] << 32) -
                     (((unsigned long long)m[5 * l + 1] + m[5 * l + 2]) << 16) + sxy(l);
            }
            if (a > 0 && b < wcy) {
                const int l = b * wcx + a - 1;
                v += ((unsigned long long)m[5 * l + 1] << 16) - sxy(l);
            }
            if (a < wcx && b > 0) {
                const int l = (b - 1) * wcx + a;
                v += ((unsigned long long)m[5 * l + 2] << 16) - sxy(l);
            }
            if (a > 0 && b > 0) v += sxy((b - 1) * wcx + a - 1);
            if (v) atomicAdd(A.rho + w.node(W, A.nx, A.ny), v * A.qmul);
        }
    }
}


// One push block: particles [base, end) of one run (end a multiple of 4 or
// the end of the padded array), window anchored at tile `anc` (-1: none).
// Thread t owns the quads base + 4t + 4k blockDim.x; the loop runs while any
// lane of the warp has a quad, so that the warp stays converged for AGG.
// !MOVE: a deposit of the particles in place; nothing is stored.
template <bool GATHER, bool DEPOSIT, bool AGG, bool MOVE = true, bool LATE = false>
__device__ __forceinline__ void push_block(const PushArgs &A, const PushGeo &G, unsigned char *smem,
                                           long long base, long long end, int anc)
{
    const Window W = setup_window(G, smem, anc);
    double *sAcc = reinterpret_cast<double *>(smem + window_bytes(G.wcx, G.wcy));
    load_window<GATHER, DEPOSIT, LATE>(G, W);
    if (threadIdx.x < 3) sAcc[threadIdx.x] = 0.0;
    __syncthreads();

    float ke = 0.f, px = 0.f, py = 0.f;
    bool bad = false;
    // byte offsets within the block's part of a field (at most 32768 particles)
    const unsigned bytes = 4u * (unsigned)(end - base), stride = 16u * blockDim.x;
    const unsigned lane16 = 16u * (threadIdx.x & 31);
    for (unsigned ow = 16u * (threadIdx.x & ~31u); ow < bytes; ow += stride) {
        const unsigned o = ow + lane16;
        const bool live = o < bytes;
        // the thread's quad of the next iteration, fetched into L2 now so
        // that its loads wait on L2 rather than DRAM (no registers held;
        // measured at 2048^2: 0.958 against 1.000 ms per launch, and
        // 0.970 ms two iterations ahead)
        if (MOVE && o + stride < bytes) {
            const unsigned on = o + stride;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(&at<char>(A.cin + base, on)));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(&at<char>(A.oxin + base, on)));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(&at<char>(A.oyin + base, on)));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(&at<char>(A.vxin + base, on)));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(&at<char>(A.vyin + base, on)));
        }
        // coherent loads (with an in-place pass the same addresses are stored below)
        int cc[4] = {-1, -1, -1, -1};
        float xo[4] = {0.f, 0.f, 0.f, 0.f}, yo[4] = {0.f, 0.f, 0.f, 0.f};
        float xv[4] = {0.f, 0.f, 0.f, 0.f}, yv[4] = {0.f, 0.f, 0.f, 0.f};
        if (live) {
            const int4 c4 = ld<LATE>(&at<int4>(A.cin + base, o));
            const float4 a4 = ld<LATE>(&at<float4>(A.oxin + base, o));
            const float4 b4 = ld<LATE>(&at<float4>(A.oyin + base, o));
            cc[0] = c4.x, cc[1] = c4.y, cc[2] = c4.z, cc[3] = c4.w;
            xo[0] = a4.x, xo[1] = a4.y, xo[2] = a4.z, xo[3] = a4.w;
            yo[0] = b4.x, yo[1] = b4.y, yo[2] = b4.z, yo[3] = b4.w;
            if (MOVE) {
                const float4 u4 = ld<LATE>(&at<float4>(A.vxin + base, o));
                const float4 v4 = ld<LATE>(&at<float4>(A.vyin + base, o));
                xv[0] = u4.x, xv[1] = u4.y, xv[2] = u4.z, xv[3] = u4.w;
                yv[0] = v4.x, yv[1] = v4.y, yv[2] = v4.z, yv[3] = v4.w;
            }
        }
        if constexpr (AGG) {
            static_assert(DEPOSIT && MOVE && !LATE, "push_grouped");
            push_grouped<GATHER>(G, W, cc, xo, yo, xv, yv, ke, px, py, bad);
        } else {
            bool whole = true;  // four cells on the grid (-1, an empty slot, is off it)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                whole = whole && (cc[j] & 0xFFFF) < G.nx && (unsigned)(cc[j] >> 16) < (unsigned)G.ny;
            if (whole)
                push_four<GATHER, DEPOSIT, MOVE, LATE>(G, W, cc, xo, yo, xv, yv, ke, px, py);
            else if (live)
                push_slots<GATHER, DEPOSIT, MOVE, LATE>(G, W, cc, xo, yo, xv, yv, ke, px, py, bad);
        }
        if (MOVE && live) store_quad<LATE>(A, base, o, cc, xo, yo, xv, yv);
    }
    // a non-finite (or overflowing) velocity makes the sum of squares non-finite
    if (MOVE) bad |= !(fabsf(ke) <= 3.0e38f);
    finish_block<DEPOSIT>(G, W, sAcc, ke, px, py, MOVE && bad);
}

}  // namespace pic
