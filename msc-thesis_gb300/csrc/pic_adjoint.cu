// pic_adjoint.cu -- discrete adjoint of the collisionless GPU step.
//
// Forward map (one charged species): v(-1/2) = v0 + c0 (q/m) F(x0) with
// c0 = -dt/2, then for n = 0..N-1: v(n+1/2) = v(n-1/2) + dt (q/m) F(x_n),
// x_(n+1) = x_n + dt v(n+1/2), where F(x)_i = sum_k w_k(x_i) E_k and
// E = S rho(x) (CIC deposit, spectral Poisson, E = -i k phi).  Objective
// J = 1/2 eps0 dA sum_k |E_k(x_N)|^2.
//
// Backward (a_x = dJ/dx, a_v = dJ/dv): a_x = grad J(x_N); for n = N-1..0:
// a_v += dt a_x (drift), then the kick transpose with mu = dt (q/m) a_v:
//   local     a_x,i += sum_k grad w_k(x_i) (E_k . mu_i)
//   scatter   g_k = sum_i w_k(x_i) mu_i                (adjoint of the gather)
//   solve     psi = S^T g, psi^ = i k.g^ / (eps0 k^2)  (S^T of the field solve)
//   gather    a_x,j += (q / dA) sum_m psi_m grad w_m(x_j) (adjoint of the deposit)
// and finally the priming kick with coefficient c0.  grad J(x_N) is the
// solve + gather with g = eps0 dA E(x_N).  The deposit's 2^-16 weight
// quantisation is not differentiated (continuous CIC weights are used).
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "pic_adjoint_dev.cuh"

namespace pic {

struct AdjArgs {
    const int32_t *cell;
    const float *ox, *oy;        // positions of the step
    float *ax, *ay;              // adjoint positions (storage order)
    const float *psi;            // S^T g
    long long n;
    int nx, ny;
    float inv_dx, inv_dy;
    float q_over_dA;
};

// Drift adjoint, kick local term and scatter of mu, one push chunk per block
// (adj_kick_block; 128^2 x 32 per cell: 16 us against 21 us with eight global
// float adds per particle).
__global__ void __launch_bounds__(256, 3)
adj_kick_kernel(KickArgs A, KickGeo K, const int32_t *anchor, int chunk, long long n4)
{
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_wait();
    pdl_trigger();
    const long long base = (long long)blockIdx.x * chunk;
    adj_kick_block<false>(A, K, smem, base, min(base + (long long)chunk, n4), anchor[blockIdx.x]);
}

// adjoint of the deposit: a_x += (q/dA) sum_m psi_m grad w_m
__global__ void __launch_bounds__(256) adj_gather_kernel(AdjArgs A)
{
    pdl_wait();
    pdl_trigger();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += stride) {
        const Cic w = cic_of(A.cell[i], A.ox[i], A.oy[i], A.nx, A.ny);
        if (!w.ok) continue;
        const float2 g = grad_dot(w, A.psi[w.i00], A.psi[w.i10], A.psi[w.i01], A.psi[w.i11],
                                  A.inv_dx, A.inv_dy);
        A.ax[i] = fmaf(A.q_over_dA, g.x, A.ax[i]);
        A.ay[i] = fmaf(A.q_over_dA, g.y, A.ay[i]);
    }
}

// psi^ = i (kx g^x + ky g^y) / (eps0 N k^2), Nyquist derivative zeroed as in
// the forward solve, zero mode removed
__global__ void __launch_bounds__(256) adj_kspace_kernel(const float2 *gh, float2 *ph, int nx, int ny,
                                                         int nh, float kx1, float ky1, float inv_eps0_n)
{
    const long long total = (long long)ny * nh;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int my = (int)idx / nh, mx = (int)idx - my * nh;  // ny nh < 2^31
        ph[idx] = adj_mode(gh[idx], gh[total + idx], mx, my, nx, ny, kx1, ky1, inv_eps0_n, idx == 0);
    }
}

__global__ void scale_planes_kernel(const float *ex, const float *ey, float s, float *gx, float *gy,
                                    long long n)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        gx[i] = s * ex[i];
        gy[i] = s * ey[i];
    }
}

// storage order -> id order (double) for two arrays
__global__ void to_id_order_kernel(const float *a, const float *b, const uint32_t *pid, long long n,
                                   double *oa, double *ob)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const uint32_t p = pid[i];
        if ((long long)p >= n) continue;
        oa[p] = a[i];
        ob[p] = b[i];
    }
}

// ---------------------------------------------------------------- driver
namespace {

// An adjoint run's device memory: one block, carved up by a layout that is
// run twice (sizes, then addresses).  Up to ADJ_STAGE_MAX bytes lie in the
// handle's stage, which later runs find in place; more, or more than the
// caller's budget for the stage (stage_fits), is allocated for the call alone.
constexpr size_t ADJ_STAGE_MAX = 256ull << 20;

struct AdjWork {
    char *base = nullptr, *own = nullptr;
    size_t used = 0;
    cufftHandle r2c2 = 0;
    ~AdjWork()
    {
        if (own) cudaFree(own);
        if (r2c2) cufftDestroy(r2c2);
    }
    template <class T> T *take(size_t n)
    {
        char *p = base + used;
        used += (n * sizeof(T) + 255) & ~(size_t)255;
        return reinterpret_cast<T *>(p);
    }
};

struct Snap {  // particle state of species 0 (storage order)
    int32_t *cell;
    float *ox, *oy, *vx, *vy;
};

Snap take_snap(AdjWork &W, size_t n)
{
    Snap S;
    S.cell = W.take<int32_t>(n);
    S.ox = W.take<float>(n);
    S.oy = W.take<float>(n);
    S.vx = W.take<float>(n);
    S.vy = W.take<float>(n);
    return S;
}

pic_status snap_copy(pic_handle *h, Snap &S, bool save, size_t n)
{
    SpeciesBuf &B = h->sp[0];
    void *live[5] = {B.cell[0], B.ox[0], B.oy[0], B.vx[0], B.vy[0]};
    void *kept[5] = {S.cell, S.ox, S.oy, S.vx, S.vy};
    for (int k = 0; k < 5; ++k)
        PIC_CUDA(cudaMemcpyAsync(save ? kept[k] : live[k], save ? live[k] : kept[k], n * 4,
                                 cudaMemcpyDeviceToDevice, h->stream));
    return PIC_OK;
}

}  // namespace

pic_status adjoint_run(pic_handle *h, const pic_init_spec *spec, long long nsteps, int every,
                       double *gx0, double *gy0, double *gvx0, double *gvy0,
                       pic_adjoint_result *out)
{
    const pic_config &c = h->cfg;
    if (c.nspecies != 1 || c.species[0].q == 0.0 || h->mcc.on || h->dsmc.on || nsteps < 1 ||
        every < 1) {
        set_error("pic_adjoint_run: needs one charged species, no collisions, nsteps >= 1, every >= 1");
        return PIC_ERR_INVALID_ARG;
    }
    if (spec) PIC_TRY(pic_init_particles(h, 0, spec));
    if (!h->fields_valid) {
        set_error("pic_adjoint_run: no particles loaded");
        return PIC_ERR_STATE;
    }
    const Geometry &g = h->g;
    SpeciesBuf &B = h->sp[0];
    cudaStream_t st = h->stream;
    const size_t np = (size_t)B.cap;
    const long long n = B.n;
    const size_t ncell = (size_t)g.nx * g.ny, nk = (size_t)g.ny * g.nh;
    const double qm = c.species[0].q / c.species[0].m, dt = c.dt;
    const int K = (int)std::min<long long>(every, nsteps);
    const int nseg = (int)((nsteps + K - 1) / K);
    AdjWork W;
    std::vector<Snap> ck(nseg - 1);  // state at the start of every segment but the last
    Snap fin = {};                   // the final state (several segments)
    std::vector<StepSlot> ring(K);   // positions and field of a segment's steps
    KickArgs A = {};
    float *gpl = nullptr, *psi = nullptr;
    float2 *gh = nullptr, *ph = nullptr;
    double *buf = nullptr;           // the gradients in id order
    DevState *saved = nullptr;
    auto layout = [&]() {
        W.used = 0;
        for (auto &S : ck) S = take_snap(W, np);
        if (nseg > 1) fin = take_snap(W, np);
        for (auto &S : ring) {
            S.cell = W.take<int32_t>(np);
            S.ox = W.take<float>(np);
            S.oy = W.take<float>(np);
            S.e = W.take<float>(2 * ncell);
        }
        A.ax = W.take<float>(np);
        A.ay = W.take<float>(np);
        A.avx = W.take<float>(np);
        A.avy = W.take<float>(np);
        gpl = W.take<float>(2 * ncell);
        psi = W.take<float>(ncell);
        gh = W.take<float2>(2 * nk);
        ph = W.take<float2>(nk);
        buf = W.take<double>(4 * (size_t)n);
        saved = W.take<DevState>(1);
    };
    layout();
    if (W.used <= ADJ_STAGE_MAX && stage_fits(h, W.used)) {
        PIC_TRY(ensure_stage(h, W.used));
        W.base = (char *)h->stage;
    } else {
        PIC_CUDA(cudaMalloc(&W.own, W.used));
        W.base = W.own;
    }
    layout();
    if (!h->spectral) {
        int dims[2] = {g.ny, g.nx};
        PIC_CUFFT(cufftPlanMany(&W.r2c2, 2, dims, nullptr, 1, (int)ncell, nullptr, 1, (int)nk,
                                CUFFT_R2C, 2));
        PIC_CUFFT(cufftSetStream(W.r2c2, st));
    }
    const StepSlot live = {B.cell[0], B.ox[0], B.oy[0], h->e};

    // The live state and field into ring slot 0, then `steps` pushes, each
    // from its slot to the next (the last one of the final segment back into
    // the live arrays): nothing is copied for the ring but its first slot.
    // (128^2 x 32 per cell, 40 steps every 10, through the torch binding: 11.0
    // ms with every slot copied, the last segment run twice, forty-odd
    // allocations and a cuFFT plan per call; 4.7 ms now.)
    auto fill_ring = [&](int steps, bool last, int adv) -> pic_status {
        PIC_CUDA(cudaMemcpyAsync(ring[0].cell, live.cell, np * 4, cudaMemcpyDeviceToDevice, st));
        PIC_CUDA(cudaMemcpyAsync(ring[0].ox, live.ox, np * 4, cudaMemcpyDeviceToDevice, st));
        PIC_CUDA(cudaMemcpyAsync(ring[0].oy, live.oy, np * 4, cudaMemcpyDeviceToDevice, st));
        PIC_CUDA(cudaMemcpyAsync(ring[0].e, live.e, 2 * ncell * 4, cudaMemcpyDeviceToDevice, st));
        for (int s = 0; s < steps; ++s) {
            const StepSlot &to = last && s == steps - 1 ? live : ring[s + 1];
            PIC_TRY(launch_push_slot(h, ring[s], to));
            PIC_TRY(record_poisson(h, adv, to.e));
        }
        return PIC_OK;
    };

    // ---- forward: prime, checkpoints every K steps, the last segment into
    // the ring, no re-sorting
    const LibrarySolve mark(h);
    if (h->mixed) {  // the field that the caller's last call left is not the library's
        PIC_TRY(deposit_now(h));
        PIC_TRY(record_poisson(h, ADV_FIELD));
    }
    PIC_TRY(pic_prime_leapfrog(h));
    if (!h->rho_clear) PIC_CUDA(cudaMemsetAsync(h->rho_fix, 0, ncell * 8, st));
    for (int m = 0; m + 1 < nseg; ++m) {
        PIC_TRY(snap_copy(h, ck[m], true, np));
        for (int s = 0; s < K; ++s) {
            PIC_TRY(record_push_all(h, 0, true, false));
            PIC_TRY(record_poisson(h, ADV_PUSH | ADV_FIELD));
        }
    }
    PIC_TRY(fill_ring((int)(nsteps - (long long)(nseg - 1) * K), true, ADV_PUSH | ADV_FIELD));
    if (nseg > 1) PIC_TRY(snap_copy(h, fin, true, np));
    h->steps_host += nsteps;
    h->since_sort += (int)std::min<long long>(nsteps, 1 << 30);
    // the diagnostics of step nsteps are kept apart from the passes below,
    // which fold nothing into the history
    PIC_CUDA(cudaMemcpyAsync(saved, h->dev, sizeof(DevState), cudaMemcpyDeviceToDevice, st));

    AdjArgs G;
    G.n = n;
    G.nx = g.nx;
    G.ny = g.ny;
    G.inv_dx = (float)(1.0 / g.dx);
    G.inv_dy = (float)(1.0 / g.dy);
    G.q_over_dA = (float)(c.species[0].q / (g.dx * g.dy));
    G.ax = A.ax;
    G.ay = A.ay;
    G.psi = psi;
    KickGeo Q;
    memset(&Q, 0, sizeof Q);
    Q.G.nx = g.nx;
    Q.G.ny = g.ny;
    Q.G.tw = g.tw;
    Q.G.th = g.th;
    Q.G.hx = Q.G.hy = g.halo;
    Q.G.wcx = g.wcx;
    Q.G.wcy = g.wcy;
    Q.gx = gpl;
    Q.gy = gpl + ncell;
    Q.inv_dx = G.inv_dx;
    Q.inv_dy = G.inv_dy;
    long long n4 = (n + 3) & ~3ll;
    const unsigned nblk = (unsigned)((n4 + B.chunk - 1) / B.chunk);
    const size_t kick_smem = kick_bytes(g.wcx, g.wcy);
    const int gp = grid_for(n, 256), gg = grid_for((long long)nk, 256);
    const float kx1 = (float)(2.0 * 3.14159265358979323846 / g.Lx);
    const float ky1 = (float)(2.0 * 3.14159265358979323846 / g.Ly);
    const float inv_eps0_n = (float)(1.0 / (c.eps0 * (double)ncell));
    // psi = S^T g (which leaves g clear) and a_x += (q/dA) sum psi grad w at
    // the positions of a slot
    auto solve_and_gather = [&](const StepSlot &S) -> pic_status {
        if (h->spectral) {
            PIC_TRY(launch_spectral_adjoint(h, gpl, gpl + ncell, gh, ph, psi));
        } else {
            PIC_CUFFT(cufftExecR2C(W.r2c2, gpl, (cufftComplex *)gh));
            adj_kspace_kernel<<<gg, 256, 0, st>>>(gh, ph, g.nx, g.ny, g.nh, kx1, ky1, inv_eps0_n);
            PIC_CUDA(cudaGetLastError());
            PIC_CUFFT(cufftExecC2R(h->plan_c2r1, (cufftComplex *)ph, psi));
            PIC_CUDA(cudaMemsetAsync(gpl, 0, 2 * ncell * 4, st));
        }
        G.cell = S.cell;
        G.ox = S.ox;
        G.oy = S.oy;
        void *args[] = {&G};
        return launch_dependent((const void *)adj_gather_kernel, gp, 256, 0, st, args);
    };
    auto kick = [&](const StepSlot &S, float C, float drift) -> pic_status {
        A.cell = S.cell;
        A.ox = S.ox;
        A.oy = S.oy;
        Q.G.ex = S.e;
        Q.G.ey = S.e + ncell;
        Q.muc = (float)(C * qm);
        Q.ddt = drift;
        if (nblk) {
            PIC_TRY(allow_dynamic_smem((const void *)adj_kick_kernel, kick_smem));
            void *args[] = {&A, &Q, &B.anchor, &B.chunk, &n4};
            PIC_TRY(launch_dependent((const void *)adj_kick_kernel, nblk, 256, kick_smem, st, args));
        }
        return solve_and_gather(S);
    };

    // ---- terminal condition: a_x = grad J(x_N)
    PIC_CUDA(cudaMemsetAsync(A.ax, 0, np * 4, st));
    PIC_CUDA(cudaMemsetAsync(A.ay, 0, np * 4, st));
    PIC_CUDA(cudaMemsetAsync(A.avx, 0, np * 4, st));
    PIC_CUDA(cudaMemsetAsync(A.avy, 0, np * 4, st));
    scale_planes_kernel<<<grid_for((long long)ncell, 256), 256, 0, st>>>(
        h->e, h->e + ncell, (float)(c.eps0 * g.dx * g.dy), gpl, gpl + ncell, (long long)ncell);
    PIC_CUDA(cudaGetLastError());
    PIC_TRY(solve_and_gather(live));

    // ---- backward over the segments, recomputing each but the last into the ring
    for (int m = nseg - 1; m >= 0; --m) {
        const int steps = (int)(std::min<long long>(nsteps, (long long)(m + 1) * K) - (long long)m * K);
        if (m < nseg - 1) {
            PIC_TRY(snap_copy(h, ck[m], false, np));
            PIC_TRY(deposit_now(h));
            PIC_TRY(record_poisson(h, 0));
            PIC_TRY(fill_ring(steps - 1, false, 0));
        }
        for (int s = steps - 1; s >= 0; --s) PIC_TRY(kick(ring[s], (float)dt, (float)dt));
    }
    // ---- the priming kick v(-1/2) = v0 - (q/m) F(x0) dt/2 (ring slot 0 of segment 0)
    PIC_TRY(kick(ring[0], (float)(-0.5 * dt), 0.f));

    // ---- outputs in id order
    to_id_order_kernel<<<gp, 256, 0, st>>>(A.ax, A.ay, B.pid[0], n, buf, buf + n);
    to_id_order_kernel<<<gp, 256, 0, st>>>(A.avx, A.avy, B.pid[0], n, buf + 2 * n, buf + 3 * n);
    PIC_CUDA(cudaGetLastError());
    // the load's derivatives need dJ/dx0, dJ/dy0 and dJ/dvx0 on the host
    std::vector<double> own;
    double *dst[4] = {gx0, gy0, gvx0, gvy0};
    if (out && spec) {
        int missing = 0;
        for (int k = 0; k < 3; ++k) missing += dst[k] ? 0 : 1;
        own.resize((size_t)missing * n);
        double *p = own.data();
        for (int k = 0; k < 3; ++k)
            if (!dst[k]) {
                dst[k] = p;
                p += n;
            }
    }
    for (int k = 0; k < 4; ++k)
        if (dst[k])
            PIC_CUDA(cudaMemcpyAsync(dst[k], buf + k * n, (size_t)n * 8, cudaMemcpyDeviceToHost, st));
    std::vector<double> dA;
    if (out && spec) {
        dA.resize(2 * (size_t)n);
        int lx = 0, ly = 0;
        if (spec->layout == PIC_LOAD_LATTICE) PIC_TRY(lattice_dims(h, n, &lx, &ly));
        PIC_TRY(launch_init_dA(h, spec, lx, ly, buf, buf + n));
        PIC_CUDA(cudaMemcpyAsync(dA.data(), buf, dA.size() * 8, cudaMemcpyDeviceToHost, st));
    }
    // ---- leave the handle at step nsteps, with the field of its own solve (as
    // a state file of these particles would)
    h->library_solve = false;
    if (nseg > 1) PIC_TRY(snap_copy(h, fin, false, np));
    if (nseg > 1 || h->mixed) {
        PIC_TRY(deposit_now(h));
        PIC_TRY(record_poisson(h, 0));
    }
    PIC_CUDA(cudaMemcpyAsync(h->dev, saved, sizeof(DevState), cudaMemcpyDeviceToDevice, st));
    pic_diag d;
    PIC_TRY(pic_diagnostics(h, &d));  // waits for all of it
    if (out) {
        out->J = d.field_energy;
        out->dJ_dbeam_v = 0.0;
        out->dJ_damp = 0.0;
        if (spec) {
            double sb = 0.0, sa = 0.0;
            for (long long i = 0; i < n; ++i) {
                sb += (i & 1) ? -dst[2][i] : dst[2][i];  // vx carries +-beam_v by id parity
                sa += dst[0][i] * dA[i] + dst[1][i] * dA[n + i];
            }
            out->dJ_dbeam_v = sb;
            out->dJ_damp = sa;
        }
    }
    return PIC_OK;
}

}  // namespace pic

extern "C" pic_status pic_adjoint_run(pic_handle *h, const pic_init_spec *spec, long long nsteps,
                                      int every, double *dJ_dx0, double *dJ_dy0, double *dJ_dvx0,
                                      double *dJ_dvy0, pic_adjoint_result *out)
{
    if (!h) {
        pic::set_error("pic_adjoint_run: null handle");
        return PIC_ERR_INVALID_ARG;
    }
    PIC_CUDA(cudaSetDevice(h->device));
    return pic::adjoint_run(h, spec, nsteps, every, dJ_dx0, dJ_dy0, dJ_dvx0, dJ_dvy0, out);
}
