// pic_collide.cu -- collision operators: electron-neutral MCC (null-collision
// method) and neutral-neutral DSMC (Bird's no-time-counter scheme).
//
// Replace (taylorj5/msc-thesis, thesisCode/):
//   mccCollisions/src/particle.cc:112-127, mccCollisions/src/pic.cu:435-466
//     Bernoulli(0.8 / 0.22) resample v = 2(u1+u2+u3-1.5), no cross sections
//   dsmcCollisions/cellTrackerAdvanced/src/main.cc:288-350, src/pic.cu:791-870
//     nearest in-cell partner, fixed probability, +-(sum of uniforms)
// with the physical operators the configuration asks for.  Random numbers
// are Philox4x32-10 (pic_internal.cuh); MCC draws per particle id and
// collision pass, DSMC per cell, pass and candidate, so both are
// reproducible for a given particle or cell whatever the storage order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "pic_internal.cuh"

namespace pic {

// ---------------------------------------------------------------- helpers
// orthonormal basis (e1, e2) perpendicular to unit u (Duff et al., "Building
// an orthonormal basis, revisited", JCGT 6(1), 2017)
__device__ __forceinline__ void perp_basis(float ux, float uy, float uz, float3 &e1, float3 &e2)
{
    const float sgn = copysignf(1.0f, uz);
    const float a = -1.0f / (sgn + uz);
    const float b = ux * uy * a;
    e1 = make_float3(1.0f + sgn * ux * ux * a, sgn * b, -sgn * ux);
    e2 = make_float3(b, sgn + uy * uy * a, -uy);
}

// unit vector at polar angle chi (cos chi = c) and azimuth 2 pi w about u
__device__ __forceinline__ float3 deflect(float ux, float uy, float uz, float c, float w)
{
    float3 e1, e2;
    perp_basis(ux, uy, uz, e1, e2);
    const float s = sqrtf(fmaxf(0.0f, 1.0f - c * c));
    float sp, cp;
    sincospif(2.0f * w, &sp, &cp);
    return make_float3(c * ux + s * (cp * e1.x + sp * e2.x), c * uy + s * (cp * e1.y + sp * e2.y),
                       c * uz + s * (cp * e1.z + sp * e2.z));
}

// ---------------------------------------------------------------- MCC
struct MccArgs {
    int32_t *ecell;
    float *eox, *eoy, *evx, *evy, *evz;
    uint32_t *epid;
    long long n0;            // electrons at the start of the pass
    long long ecap;
    int32_t *icell;
    float *iox, *ioy, *ivx, *ivy, *ivz;
    uint32_t *ipid;
    long long ni0;           // ions at the start of the pass
    long long icap;
    int has_ion;
    const float *tab;   // [energy | elastic | excitation | ionisation] x ntab
    int ntab;
    float ln_emin, inv_dln;
    float half_me_over_e;  // E[eV] = half_me_over_e * |v|^2
    float ng, nu_max, two_m_over_M;
    uint32_t cand_below;  // candidate when the draw's top 24 bits are below (u01f < P_null)
    float e_exc, e_ion, vth_ion;
    uint32_t k0, k1;
    int e, i;             // electron and ion species
    DevState *dev;
};

__device__ __forceinline__ void mcc_sigmas(const MccArgs &A, const float *tab, float E,
                                           float &sel, float &sexc, float &sion)
{
    const int nt = A.ntab;
    int k;
    float f;
    if (E <= tab[0]) {
        k = 0;
        f = 0.f;
    } else if (E >= tab[nt - 1]) {
        k = nt - 2;
        f = 1.f;
    } else {
        k = (int)((__logf(E) - A.ln_emin) * A.inv_dln);
        k = min(max(k, 0), nt - 2);
        // the log index can be off by one near a table point; fix it exactly
        if (E < tab[k]) k = max(k - 1, 0);
        if (E >= tab[k + 1]) k = min(k + 1, nt - 2);
        f = (E - tab[k]) / (tab[k + 1] - tab[k]);
    }
    const float *el = tab + nt, *ex = tab + 2 * nt, *io = tab + 3 * nt;
    sel = fmaf(f, el[k + 1] - el[k], el[k]);
    sexc = fmaf(f, ex[k + 1] - ex[k], ex[k]);
    sion = fmaf(f, io[k + 1] - io[k], io[k]);
}

constexpr int MCC_THREADS = 256;
constexpr int MCC_BLOCKS_PER_SM = 4;
constexpr int MCC_PER_LANE = 8;
constexpr int MCC_CHUNK = 32 * MCC_PER_LANE;  // electrons a warp tests at a time
constexpr int MCC_QUEUE = MCC_CHUNK + 32;     // a warp's candidates: a chunk's and up to 31 carried over

// Collision of candidate electron i (r: its first draw of this pass):
// real (elastic, excitation, ionisation with ion birth) or null.
__device__ __forceinline__ void mcc_collide(const MccArgs &A, const float *s_tab, long long i,
                                            uint32_t pid, unsigned long long pass, const U4 &r,
                                            unsigned &c_el, unsigned &c_exc, unsigned &c_ion,
                                            unsigned &c_null, bool &overflow)
{
    float vx = A.evx[i], vy = A.evy[i], vz = A.evz[i];
    const float v2 = vx * vx + vy * vy + vz * vz;
    const float v = sqrtf(v2);
    const float E = A.half_me_over_e * v2;
    float sel, sexc, sion;
    mcc_sigmas(A, s_tab, E, sel, sexc, sion);
    if (E < A.e_exc) sexc = 0.f;
    if (E < A.e_ion) sion = 0.f;
    const float nu_el = A.ng * sel * v, nu_exc = A.ng * sexc * v, nu_ion = A.ng * sion * v;
    const float R = u01f(r.y) * A.nu_max;
    const float ux = v > 0.f ? vx / v : 0.f, uy = v > 0.f ? vy / v : 0.f;
    const float uz = v > 0.f ? vz / v : 1.f;
    if (R < nu_el) {
        const float c = 1.f - 2.f * u01f(r.z);
        const float En = E * (1.f - A.two_m_over_M * (1.f - c));
        const float3 d = deflect(ux, uy, uz, c, u01f(r.w));
        const float vn = sqrtf(En / A.half_me_over_e);
        vx = vn * d.x;
        vy = vn * d.y;
        vz = vn * d.z;
        ++c_el;
    } else if (R < nu_el + nu_exc) {
        const float c = 1.f - 2.f * u01f(r.z);
        const float3 d = deflect(ux, uy, uz, c, u01f(r.w));
        const float vn = sqrtf(fmaxf(E - A.e_exc, 0.f) / A.half_me_over_e);
        vx = vn * d.x;
        vy = vn * d.y;
        vz = vn * d.z;
        ++c_exc;
    } else if (R < nu_el + nu_exc + nu_ion) {
        const U4 r2 = philox4x32_10(U4{pid, (uint32_t)pass, 1u, STREAM_MCC}, A.k0, A.k1);
        const float Er = fmaxf(E - A.e_ion, 0.f);
        const float Ej = u01f(r2.x) * Er, Es = Er - Ej;
        const float3 ds = deflect(ux, uy, uz, 1.f - 2.f * u01f(r.z), u01f(r.w));
        const float3 dj = deflect(ux, uy, uz, 1.f - 2.f * u01f(r2.y), u01f(r2.z));
        const float vs = sqrtf(Es / A.half_me_over_e), vj = sqrtf(Ej / A.half_me_over_e);
        vx = vs * ds.x;
        vy = vs * ds.y;
        vz = vs * ds.z;
        ++c_ion;
        if (A.has_ion) {
            // reserve the ion slot, then the electron slot; a reservation past
            // the capacity is given back, so the successful slots stay
            // contiguous from the old count
            const long long ji = A.ni0 + (long long)atomicAdd(&A.dev->born[1], 1ull);
            long long je = A.ecap;
            if (ji < A.icap) je = A.n0 + (long long)atomicAdd(&A.dev->born[0], 1ull);
            if (ji < A.icap && je < A.ecap) {
                A.ecell[je] = A.ecell[i];
                A.eox[je] = A.eox[i];
                A.eoy[je] = A.eoy[i];
                A.evx[je] = vj * dj.x;
                A.evy[je] = vj * dj.y;
                A.evz[je] = vj * dj.z;
                A.epid[je] = (uint32_t)je;
                const U4 r3 = philox4x32_10(U4{pid, (uint32_t)pass, 2u, STREAM_MCC}, A.k0, A.k1);
                const float ra = sqrtf(-2.f * __logf(u01f(r3.x))), rb = sqrtf(-2.f * __logf(u01f(r3.z)));
                float sa, ca, sb, cb;
                sincospif(2.f * u01f(r3.y), &sa, &ca);
                sincospif(2.f * u01f(r3.w), &sb, &cb);
                A.icell[ji] = A.ecell[i];
                A.iox[ji] = A.eox[i];
                A.ioy[ji] = A.eoy[i];
                A.ivx[ji] = A.vth_ion * ra * ca;
                A.ivy[ji] = A.vth_ion * ra * sa;
                A.ivz[ji] = A.vth_ion * rb * cb;
                A.ipid[ji] = (uint32_t)ji;
            } else {
                // no room: give back what was reserved and report; an ion slot
                // whose electron did not fit stays empty (cell -1)
                if (ji >= A.icap) {
                    atomicAdd(&A.dev->born[1], (unsigned long long)-1ll);
                } else {
                    atomicAdd(&A.dev->born[0], (unsigned long long)-1ll);
                    A.icell[ji] = -1;
                    A.ipid[ji] = (uint32_t)ji;
                }
                overflow = true;
            }
        }
    } else {
        ++c_null;
        return;
    }
    A.evx[i] = vx;
    A.evy[i] = vy;
    A.evz[i] = vz;
}

// One null-collision pass over the electrons present at its start (births
// are counted apart and added to the species' counts by the last block).
// Each warp works on its own, without block barriers: it tests MCC_CHUNK
// electrons at a time (one Philox draw per electron, keyed by particle id and
// pass; the ids of its next chunk are loaded meanwhile), queues the
// candidates (fraction P_null, a few percent) in shared memory and collides
// them 32 at a time, so that the costly collision path runs in full warps
// and one warp's collisions overlap the other warps' draws.  Bound by the
// Philox arithmetic (about 60 issue slots per electron, 32 us for 16.8 M);
// whether a slot is live is looked up for candidates only.  512^2 x 64 per
// cell: 79 us against 117 us with a block-wide queue (a barrier before and
// after each chunk's collisions, which half the threads sat out).
__global__ void __launch_bounds__(MCC_THREADS, MCC_BLOCKS_PER_SM) mcc_kernel(MccArgs A)
{
    extern __shared__ float s_tab[];  // 4 ntab table floats, then a candidate queue per warp
    for (int i = threadIdx.x; i < 4 * A.ntab; i += blockDim.x) s_tab[i] = A.tab[i];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint32_t *q = reinterpret_cast<uint32_t *>(s_tab + 4 * A.ntab) + MCC_QUEUE * (threadIdx.x >> 5);
    A.n0 = min(A.dev->n[A.e], A.ecap);
    A.ni0 = A.has_ion ? A.dev->n[A.i] : 0;
    const unsigned long long pass = A.dev->mcc_pass + 1ull;
    unsigned c_el = 0, c_exc = 0, c_ion = 0, c_null = 0;
    bool overflow = false;
    const uint32_t n = (uint32_t)A.n0;  // capacities are below 2^31
    const uint32_t stride = gridDim.x * (MCC_THREADS / 32) * MCC_CHUNK;
    uint32_t c0 = (blockIdx.x * (MCC_THREADS / 32) + (threadIdx.x >> 5)) * MCC_CHUNK;
    uint32_t pid[MCC_PER_LANE];
    auto load = [&](uint32_t base) {
#pragma unroll
        for (int j = 0; j < MCC_PER_LANE; ++j) {
            const uint32_t i = base + j * 32 + lane;
            pid[j] = i < n ? A.epid[i] : 0u;
        }
    };
    auto collide = [&](uint32_t i) {
        if (A.ecell[i] < 0) return;  // an empty slot
        const uint32_t id = A.epid[i];
        const U4 r = philox4x32_10(U4{id, (uint32_t)pass, 0u, STREAM_MCC}, A.k0, A.k1);
        mcc_collide(A, s_tab, i, id, pass, r, c_el, c_exc, c_ion, c_null, overflow);
    };
    int nq = 0;  // queued candidates (warp-uniform)
    if (c0 < n) load(c0);
    for (; c0 < n; c0 += stride) {
        unsigned cand = 0u;
#pragma unroll
        for (int j = 0; j < MCC_PER_LANE; ++j) {
            const U4 r = philox4x32_10(U4{pid[j], (uint32_t)pass, 0u, STREAM_MCC}, A.k0, A.k1);
            if ((r.x >> 8) < A.cand_below && c0 + j * 32 + lane < n) cand |= 1u << j;
        }
        if (n - c0 > stride) load(c0 + stride);
#pragma unroll
        for (int j = 0; j < MCC_PER_LANE; ++j) {
            const bool mine = (cand >> j) & 1u;
            const unsigned m = __ballot_sync(full, mine);
            if (mine) q[nq + __popc(m & ((1u << lane) - 1u))] = c0 + j * 32 + lane;
            nq += __popc(m);
        }
        __syncwarp();
        while (nq >= 32) {
            nq -= 32;
            collide(q[nq + lane]);
        }
        __syncwarp();  // the queue is written again by the next chunk
    }
    if (lane < nq) collide(q[lane]);
    c_el = __reduce_add_sync(full, c_el);
    c_exc = __reduce_add_sync(full, c_exc);
    c_ion = __reduce_add_sync(full, c_ion);
    c_null = __reduce_add_sync(full, c_null);
    if (lane < 4) {
        const unsigned c = lane == 0 ? c_el : lane == 1 ? c_exc : lane == 2 ? c_ion : c_null;
        if (c) atomicAdd(&A.dev->coll[lane][acc_slot()], (unsigned long long)c);
    }
    const int any_over = __syncthreads_or(overflow ? 1 : 0);
    if (threadIdx.x == 0) {
        if (any_over) atomicOr(&A.dev->err, (unsigned)PIC_DEVERR_CAPACITY);
        __threadfence();  // this block's births before its ticket
        if (atomicInc(&A.dev->ticket, gridDim.x - 1) == gridDim.x - 1) {
            __threadfence();
            A.dev->n[A.e] += (long long)atomicExch(&A.dev->born[0], 0ull);
            if (A.has_ion) A.dev->n[A.i] += (long long)atomicExch(&A.dev->born[1], 0ull);
            A.dev->mcc_pass = pass;
        }
    }
}

// ---------------------------------------------------------------- DSMC
struct NtcArgs {
    float *vx, *vy, *vz;      // the species' sorted buffer
    const uint32_t *offset;   // per key: particles [offset[k], offset[k+1])
    float *sgmax;             // per key (sigma g)_max
    long long nkeys;
    long long nslots;         // slots of the sorted buffer (bound of the offsets)
    float sigma;              // pi d^2
    float coef;               // F_N dt_c / (2 V_c)
    uint32_t k0, k1;
    DevState *dev;
};

__global__ void __launch_bounds__(256) ntc_kernel(NtcArgs A)
{
    __shared__ unsigned long long s_cnt[2];
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0ull;
    __syncthreads();
    const unsigned long long pass = A.dev->dsmc_pass;
    unsigned ncoll = 0, ncand = 0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long key = (long long)blockIdx.x * blockDim.x + threadIdx.x; key < A.nkeys;
         key += stride) {
        const uint32_t o0 = A.offset[key], o1 = A.offset[key + 1];
        if (o1 < o0 || (long long)o1 > A.nslots) {  // offsets that do not fit the slots
            atomicOr(&A.dev->err, (unsigned)PIC_DEVERR_SORT);
            continue;
        }
        const uint32_t n = o1 - o0;
        if (n < 2) continue;
        float sgm = A.sgmax[key];
        const float want = A.coef * (float)n * (float)(n - 1) * sgm;
        const U4 r0 = philox4x32_10(U4{(uint32_t)key, (uint32_t)pass, 0u, STREAM_DSMC}, A.k0, A.k1);
        const float fl = floorf(want);
        const uint32_t nc = (uint32_t)fl + (u01f(r0.x) < want - fl ? 1u : 0u);
        for (uint32_t c = 0; c < nc; ++c) {
            const U4 r = philox4x32_10(U4{(uint32_t)key, (uint32_t)pass, 2u * c + 1u, STREAM_DSMC},
                                       A.k0, A.k1);
            uint32_t a = min((uint32_t)(u01f(r.x) * (float)n), n - 1);
            uint32_t b = min((uint32_t)(u01f(r.y) * (float)(n - 1)), n - 2);
            if (b >= a) ++b;
            const uint32_t i = o0 + a, j = o0 + b;
            const float gx = A.vx[i] - A.vx[j], gy = A.vy[i] - A.vy[j], gz = A.vz[i] - A.vz[j];
            const float g = sqrtf(gx * gx + gy * gy + gz * gz);
            const float sg = A.sigma * g;
            if (sg > sgm) sgm = sg;
            ++ncand;
            if (u01f(r.z) * sgm >= sg) continue;
            // hard spheres: isotropic post-collision relative velocity in the CM frame
            const U4 r2 = philox4x32_10(U4{(uint32_t)key, (uint32_t)pass, 2u * c + 2u, STREAM_DSMC},
                                        A.k0, A.k1);
            const float cx = 2.f * u01f(r.w) - 1.f;
            const float sx = sqrtf(fmaxf(0.f, 1.f - cx * cx));
            float sp, cp;
            sincospif(2.f * u01f(r2.x), &sp, &cp);
            const float hx = 0.5f * g * cx, hy = 0.5f * g * sx * cp, hz = 0.5f * g * sx * sp;
            const float mx = 0.5f * (A.vx[i] + A.vx[j]), my = 0.5f * (A.vy[i] + A.vy[j]);
            const float mz = 0.5f * (A.vz[i] + A.vz[j]);
            A.vx[i] = mx + hx;
            A.vy[i] = my + hy;
            A.vz[i] = mz + hz;
            A.vx[j] = mx - hx;
            A.vy[j] = my - hy;
            A.vz[j] = mz - hz;
            ++ncoll;
        }
        A.sgmax[key] = sgm;
    }
    atomicAdd(&s_cnt[0], (unsigned long long)ncoll);
    atomicAdd(&s_cnt[1], (unsigned long long)ncand);
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&A.dev->coll[4][acc_slot()], s_cnt[0]);
        atomicAdd(&A.dev->coll[5][acc_slot()], s_cnt[1]);
    }
}

__global__ void bump_kernel(unsigned long long *counter) { *counter += 1ull; }

// ---------------------------------------------------------------- launchers
// The number of 24-bit draws k with u01f(k << 8) < p (u01f is monotone): an
// electron is a candidate when its draw's top 24 bits are below it.
uint32_t mcc_candidates_below(float p)
{
    uint32_t lo = 0, hi = 1u << 24;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) / 2;
        if (u01f(mid << 8) < p)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

pic_status launch_mcc(pic_handle *h)
{
    const MccState &M = h->mcc;
    SpeciesBuf &E = h->sp[M.e];
    MccArgs A;
    memset(&A, 0, sizeof A);
    A.ecell = E.cell[0];
    A.eox = E.ox[0];
    A.eoy = E.oy[0];
    A.evx = E.vx[0];
    A.evy = E.vy[0];
    A.evz = E.vz[0];
    A.epid = E.pid[0];
    A.ecap = E.cap;
    if (M.i >= 0) {
        SpeciesBuf &I = h->sp[M.i];
        A.icell = I.cell[0];
        A.iox = I.ox[0];
        A.ioy = I.oy[0];
        A.ivx = I.vx[0];
        A.ivy = I.vy[0];
        A.ivz = I.vz[0];
        A.ipid = I.pid[0];
        A.icap = I.cap;
        A.has_ion = 1;
    }
    A.tab = M.tab;
    A.ntab = M.ntab;
    A.ln_emin = M.ln_emin;
    A.inv_dln = M.inv_dln;
    A.half_me_over_e = M.half_me_over_e;
    A.ng = M.ng;
    A.nu_max = M.nu_max;
    A.cand_below = M.cand_below;
    A.e = M.e;
    A.i = M.i;
    A.two_m_over_M = M.two_m_over_M;
    A.e_exc = M.e_exc;
    A.e_ion = M.e_ion;
    A.vth_ion = M.vth_ion;
    A.k0 = (uint32_t)M.seed;
    A.k1 = (uint32_t)(M.seed >> 32);
    A.dev = h->dev;
    void *args[] = {&A};
    const long long warps = (E.cap + MCC_CHUNK - 1) / MCC_CHUNK, per = MCC_THREADS / 32;
    const long long most = (long long)MCC_BLOCKS_PER_SM * device_sms();
    const unsigned blocks = (unsigned)std::max(1ll, std::min((warps + per - 1) / per, most));
    const size_t smem = 4 * M.ntab * sizeof(float) + (MCC_THREADS / 32) * MCC_QUEUE * sizeof(uint32_t);
    PIC_TRY(allow_dynamic_smem((const void *)mcc_kernel, smem));
    return launch_dependent((const void *)mcc_kernel, blocks, MCC_THREADS, smem, h->stream, args);
}

// DSMC pass on species D.s, which must have just been sorted (buffer 1, offsets)
pic_status launch_ntc(pic_handle *h)
{
    const DsmcState &D = h->dsmc;
    SpeciesBuf &B = h->sp[D.s];
    NtcArgs A;
    A.vx = B.vx[1];
    A.vy = B.vy[1];
    A.vz = B.vz[1];
    A.offset = h->offset;
    A.sgmax = D.sgmax;
    A.nkeys = (long long)h->g.nx * h->g.ny;
    A.nslots = B.cap;
    A.sigma = D.sigma;
    A.coef = D.coef;
    A.k0 = (uint32_t)D.seed;
    A.k1 = (uint32_t)(D.seed >> 32);
    A.dev = h->dev;
    ntc_kernel<<<grid_for(A.nkeys, 256), 256, 0, h->stream>>>(A);
    PIC_CUDA(cudaGetLastError());
    bump_kernel<<<1, 1, 0, h->stream>>>(&h->dev->dsmc_pass);
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

}  // namespace pic
