"""What a program that uses this library has it do, as cases that can be timed.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call, run() is one pass through the
public entry points, work() the bytes and operations a pass cannot do
without, and exact() the same outputs in 64 bits from plain torch.

Physics cases return what a run is for: the particles' state by particle id
(cell-unit positions and velocities, single precision as the library holds
them) and the field-energy history of the pass.  Plasma units (eps0 = 1,
omega_pe = 1) unless a case collides.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "msc-thesis_gb300"))

import picgpu as P  # noqa: E402

TWO_PI = 2.0 * math.pi
E_CH, M_E, K_B, EPS0 = 1.602176634e-19, 9.1093837015e-31, 1.380649e-23, 8.8541878128e-12
M_I, M_GAS, D_GAS = 73000.0 * M_E, 6.6e-26, 3.6e-10
N_GAS, T_GAS = 3.2e21, 300.0

# loads above this are made on the device, as a program of that size does
HOST_LOAD_MAX = 1 << 24
# exact() stops above this many particle-steps (its share of 20 seconds)
EXACT_MAX = 400_000_000


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the library driven stage by stage, as the reference's own loop calls
        # it, on the smallest grid of the batched configuration: all latency
        dict(name="staged_64x64", kind="staged", load="two_stream", nx=64, ny=64,
             particles=64 * 64 * 16, steps=20),
        # two-stream instability, 128 x 128, 100 electrons per cell, dt 0.1
        dict(name="step_two_stream_128x128", kind="step", load="two_stream", nx=128, ny=128,
             particles=128 * 128 * 100, steps=100),
        # sides that are no powers of two, a particle count that fills no block
        dict(name="step_landau_250x180", kind="step", load="landau", nx=250, ny=180,
             particles=250 * 180 * 23 + 17, steps=60),
        # Landau damping, 2048 x 2048, 32 electrons per cell: the headline
        # configuration with the push chunk its autotuner picks
        dict(name="step_landau_2048x2048", kind="step", load="landau", nx=2048, ny=2048,
             particles=2048 * 2048 * 32, steps=100, chunk=16384),
        # host arrays in, a run, host arrays out, in one call on page-locked memory
        dict(name="run_host_512x512", kind="run_host", load="landau", nx=512, ny=512,
             particles=512 * 512 * 32, steps=20),
        # electrons and ions with null-collision MCC, 512 x 512, 64 + 64 per cell
        dict(name="mcc_512x512", kind="mcc", nx=512, ny=512, electrons=64, neutrals=0, steps=60),
        # the same with 50 hard-sphere neutrals per cell and DSMC every step
        dict(name="dsmc_512x512", kind="mcc", nx=512, ny=512, electrons=64, neutrals=50, steps=40),
        # a batch of independent two-stream runs, uneven grids and densities
        dict(name="ensemble_16", kind="ensemble", runs=16, mix=0, side=512, ppc=256, steps=40),
        # gradients of the final field energy through the torch binding
        dict(name="adjoint_128x128", kind="adjoint", load="two_stream", nx=128, ny=128,
             particles=128 * 128 * 32, steps=40, every=10),
        # every run's gradients of a batch
        dict(name="ensemble_adjoint_8", kind="ensemble_adjoint", runs=8, mix=1, side=256, ppc=64,
             steps=50, every=25),
        # the reference's one call, on its default grid
        dict(name="compat_run_32x32", kind="compat_run", nx=32, ny=32, npx=40, npy=40, dim=10,
             steps=200),
        # the reference's conventions on the two-stream configuration's size, FP64
        dict(name="compat_steps_128x128", kind="compat_steps", nx=128, ny=128, npx=1280, npy=1280,
             dim=10, steps=40),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(v):
    """The next size from v on whose prime factors are 2, 3, 5 and 7."""
    r = v
    for p in (2, 3, 5, 7):
        while r % p == 0:
            r //= p
    return v if r == 1 else _smooth(v + 1)


def _grid(rng, lo, hi):
    """Two sides between lo and hi: powers of two half of the time, else sizes that
    transform well (the library needs divisors for its tiles: it refuses many
    others), odd ones among them."""
    if rng.random() < 0.5:
        return tuple(1 << int(round(math.log2(_spread(rng, lo, hi)))) for _ in range(2))
    return tuple(_smooth(_spread(rng, lo, min(hi, 700))) for _ in range(2))


def draw(rng):
    kind = rng.choice(["staged", "step", "step", "step", "run_host", "mcc", "mcc", "ensemble",
                       "ensemble", "adjoint", "ensemble_adjoint", "compat_run", "compat_steps"])
    load = rng.choice(["two_stream", "landau"])
    if kind == "staged":
        nx, ny = _grid(rng, 32, 256)
        return dict(kind=kind, load=load, nx=nx, ny=ny,
                    particles=nx * ny * _spread(rng, 10, 64) + rng.randrange(4), steps=rng.randint(5, 20))
    if kind == "step":
        nx, ny = _grid(rng, 32, 2048)
        ppc = min(_spread(rng, 10, 128), max(10, (1 << 27) // (nx * ny)))
        n = nx * ny * ppc + rng.randrange(4)
        return dict(kind=kind, load=load, nx=nx, ny=ny, particles=n,
                    steps=rng.randint(20, 100 if n < 1 << 25 else 60),
                    chunk=rng.choice([0, 0, 4096, 16384 if ppc >= 32 else 0]))
    if kind == "run_host":
        nx, ny = _grid(rng, 128, 1024)
        n = nx * ny * min(_spread(rng, 10, 64), (1 << 24) // (nx * ny)) + rng.randrange(4)
        return dict(kind=kind, load=load, nx=nx, ny=ny, particles=n, steps=rng.randint(5, 40))
    if kind == "mcc":
        nx, ny = _grid(rng, 64, 512)
        return dict(kind=kind, nx=nx, ny=ny, electrons=_spread(rng, 10, 64),
                    neutrals=rng.choice([0, _spread(rng, 8, 50)]), steps=rng.randint(20, 40))
    if kind == "ensemble":
        return dict(kind=kind, runs=rng.randint(3, 24), mix=rng.randrange(1000),
                    side=rng.choice([64, 128, 256]), ppc=rng.choice([32, 64, 256]),
                    steps=rng.randint(20, 60))
    if kind == "adjoint":
        nx, ny = _grid(rng, 32, 192)
        steps = rng.randint(10, 40)
        return dict(kind=kind, load=load, nx=nx, ny=ny,
                    particles=nx * ny * _spread(rng, 10, 32) + rng.randrange(4), steps=steps,
                    every=rng.randint(5, steps))
    if kind == "ensemble_adjoint":
        steps = rng.randint(10, 50)
        return dict(kind=kind, runs=rng.randint(2, 10), mix=rng.randrange(1000),
                    side=rng.choice([64, 128, 256]), ppc=rng.choice([16, 32, 64]), steps=steps,
                    every=rng.randint(5, steps))
    nx, ny = _grid(rng, 16, 192)
    if kind == "compat_run":
        return dict(kind=kind, nx=nx, ny=ny, npx=_spread(rng, 10, 200), npy=_spread(rng, 10, 200),
                    dim=rng.choice([10, 13, 20]), steps=rng.randint(20, 200))
    return dict(kind=kind, nx=nx, ny=ny, npx=_spread(rng, 100, 1280), npy=_spread(rng, 100, 1280),
                dim=rng.choice([10, 13, 20]), steps=rng.randint(10, 40))


# ------------------------------------------------------------------ loads
def _generator(seed, stream):
    g = torch.Generator("cuda")
    g.manual_seed(1000003 * int(seed) + stream)
    return g


def _domain(case):
    if case["load"] == "two_stream":
        return 4.0 * math.pi, 4.0 * math.pi, 0.1
    return 0.05 * case["nx"], 0.05 * case["ny"], 0.05


def _plasma(case, seed):
    """x, y, vx, vy (64 bits, on the GPU): two beams at +-0.2 with a displacement
    of 1e-3 in mode 1, or a Maxwellian with a density wave of 1 % in mode (1, 1)."""
    Lx, Ly, _ = _domain(case)
    n, g = case["particles"], _generator(seed, 0)
    x = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * Lx
    y = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * Ly
    vx = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    vy = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    if case["load"] == "two_stream":
        x = x + 1e-3 * torch.cos(TWO_PI / Lx * x)
        beam = 1.0 - 2.0 * (torch.arange(n, device="cuda") % 2)
        vx, vy = 0.2 * beam + 0.01 * vx, 0.01 * vy
    else:
        kx, ky = TWO_PI / Lx, TWO_PI / Ly
        s = torch.sin(kx * x + ky * y) * (0.01 / (kx * kx + ky * ky))
        x, y = x - kx * s, y - ky * s
        vx, vy = 0.05 * vx, 0.05 * vy
    return torch.remainder(x, Lx), torch.remainder(y, Ly), vx, vy


def _spec(case, seed):
    """The same two loads made by the library on the device."""
    n = case["particles"]
    if case["load"] == "two_stream":
        return P.init_spec(n, vth=(0.01, 0.01, 0.0), beam_v=0.2, pert_kind=P.PERT_XDISP,
                           pert_amp=1e-3, pert_mx=1, seed=seed)
    return P.init_spec(n, vth=(0.05, 0.05, 0.0), pert_kind=P.PERT_DENSITY, pert_amp=0.01,
                       pert_mx=1, pert_my=1, seed=seed)


def _electrons(case):
    """A handle for one electron species of unit plasma frequency."""
    Lx, Ly, dt = _domain(case)
    n, A = case["particles"], Lx * Ly
    return P.Handle(P.config(case["nx"], case["ny"], Lx, Ly, dt, [P.species(n, -A / n, A / n, -1)],
                             chunk=case.get("chunk", 0)))


def _host(arrays):
    return [a.cpu().numpy() for a in arrays]


def _cross_sections():
    """Elastic 5e-20 m^2; excitation from 11.5 eV to 2e-20 at 30 eV, ionisation
    from 15.8 eV to 3e-20 at 100 eV, each linear and then flat."""
    e = 0.01 * 1e5 ** (np.arange(256) / 255.0)
    return (np.full(256, 5e-20), 2e-20 * np.clip((e - 11.5) / 18.5, 0.0, 1.0),
            3e-20 * np.clip((e - 15.8) / 84.2, 0.0, 1.0))


def _discharge(case, seed):
    """Electrons (2 eV) and ions against a neutral background, and with neutrals
    a bimodal 300 K / 1000 K hard-sphere gas, loaded and primed."""
    nx, ny = case["nx"], case["ny"]
    Lx, Ly = 2e-4 * nx, 2e-4 * ny
    ne, nn = nx * ny * case["electrons"], nx * ny * case["neutrals"]
    w = 1e15 * Lx * Ly / ne
    sp = [P.species(ne + ne // 4, -E_CH * w, M_E * w, -1, P.SPECIES_HAS_VZ),
          P.species(ne + ne // 4, E_CH * w, M_I * w, 1, P.SPECIES_HAS_VZ)]
    wn = N_GAS * Lx * Ly / max(nn, 1)
    if nn:
        sp.append(P.species(nn, 0.0, M_GAS * wn, 0, P.SPECIES_HAS_VZ))
    h = P.Handle(P.config(nx, ny, Lx, Ly, 1e-11, sp, eps0=EPS0, sort_every=40))
    gas_eV = K_B * T_GAS / E_CH
    ve, vi = math.sqrt(2.0 * E_CH / M_E), math.sqrt(K_B * T_GAS / M_I)
    h.init_particles(0, P.init_spec(ne, vth=(ve, ve, ve), seed=3 * seed))
    h.init_particles(1, P.init_spec(ne, vth=(vi, vi, vi), seed=3 * seed + 1))
    h.set_mcc(0, 1, N_GAS, gas_eV, M_E, M_I, E_CH, 0.01, 1000.0, *_cross_sections(), 11.5, 15.8,
              seed)
    if nn:
        g = _generator(seed, 1)
        xy = torch.rand((2, nn), generator=g, device="cuda", dtype=torch.float64)
        s = torch.where(torch.arange(nn, device="cuda") % 2 == 0, math.sqrt(K_B * 300.0 / M_GAS),
                        math.sqrt(K_B * 1000.0 / M_GAS))
        v = torch.randn((3, nn), generator=g, device="cuda", dtype=torch.float64) * s
        h.set_particles(2, *_host([xy[0] * Lx, xy[1] * Ly, v[0], v[1], v[2]]))
        h.set_dsmc(2, D_GAS, wn, 1.0, math.pi * D_GAS ** 2 * 3000.0, seed)
    h.prime_leapfrog()
    return h, [ne, ne] + [nn] * bool(nn)


def _batch(case):
    """(side, particles per cell, drift, amplitude) of every run of a batch."""
    rng = np.random.default_rng(case["mix"])
    sides = [s for s in (64, 128, 256, 512) if s <= case["side"]]
    ppcs = [p for p in (16, 32, 64, 128, 256) if p <= case["ppc"]]
    r = case["runs"]
    return list(zip(rng.choice(sides, r).tolist(), rng.choice(ppcs, r).tolist(),
                    rng.uniform(0.1, 0.3, r).tolist(),
                    np.exp(rng.uniform(math.log(1e-4), math.log(1e-2), r)).tolist()))


def _ensemble(case, seed):
    L, cfgs, specs = 4.0 * math.pi, [], []
    for r, (side, ppc, drift, amp) in enumerate(_batch(case)):
        n = side * side * ppc
        cfgs.append(P.config(side, side, L, L, 0.1, [P.species(n, -L * L / n, L * L / n, -1)]))
        specs.append(P.init_spec(n, vth=(0.01, 0.01, 0.0), beam_v=drift, pert_kind=P.PERT_XDISP,
                                 pert_amp=amp, pert_mx=1, seed=1000 * seed + r))
    cfgs[0].chunk, cfgs[0].sort_every = 4096, 20  # what the ensemble's autotuner picks
    return P.Ensemble(cfgs), specs


def _compat(case, seed):
    """The reference's parameters, and positions and velocities as its program holds them."""
    p = P.ref_params(xDim=case["dim"], yDim=case["dim"], nx=case["nx"], ny=case["ny"],
                     npx=case["npx"], npy=case["npy"], dt=0.01, tmax=0.01 * (case["steps"] - 0.5))
    rng = np.random.default_rng(seed)
    n = case["npx"] * case["npy"]
    xy = rng.uniform(0.0, case["dim"], (2, n))
    v = rng.normal(0.0, 1.0, (2, n))
    return p, (xy[0], xy[1], v[0], v[1])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("staged", "step", "run_host", "adjoint"):
        h = _electrons(case)
        s = dict(kind=kind, case=case, handle=h, counts=[case["particles"]], at=0)
        if kind == "run_host":
            s["arrays"] = [a.cpu().pin_memory().numpy() for a in _plasma(case, seed)]
            s["out"] = [torch.empty(case["particles"], dtype=torch.float64, pin_memory=True).numpy()
                        for _ in range(4)]
        elif kind == "adjoint":
            s["leaves"] = [a.requires_grad_() for a in _plasma(case, seed)]
            s["energy"] = P.field_energy_function(h, case["steps"], case["every"])
        else:
            if case["particles"] > HOST_LOAD_MAX:
                h.init_particles(0, _spec(case, seed))
            else:
                h.set_particles(0, *_host(_plasma(case, seed)))
            h.prime_leapfrog()
            h.synchronize()
        return s
    if kind == "mcc":
        h, counts = _discharge(case, seed)
        h.synchronize()
        return dict(kind="step", case=case, handle=h, counts=counts, at=0)
    if kind in ("ensemble", "ensemble_adjoint"):
        e, specs = _ensemble(case, seed)
        if kind == "ensemble":
            e.init(specs)
        return dict(kind=kind, case=case, ensemble=e, specs=specs, at=0)
    p, arrays = _compat(case, seed)
    return dict(kind=kind, case=case, params=p, arrays=arrays)


# ------------------------------------------------------------------ one pass
class _DeviceArray:
    """A borrowed device array for torch.as_tensor."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=3)


def _by_id(h, species, count, loaded, vz):
    """Rows (x, y in cells, velocity) of the particles loaded at the start, by id, on
    the GPU.  (Particles born since have ids in the order in which the GPU's
    blocks came to them; they are counted and left out.)"""
    v = h.particles_device(species)

    def view(p, typestr):
        return torch.as_tensor(_DeviceArray(p, count, typestr), device="cuda")

    cell, pid = view(v.cell_dev, "<i4"), view(v.pid_dev, "<i4")
    cols = [(cell & 0xFFFF) + view(v.ox_dev, "<f4"), (cell >> 16) + view(v.oy_dev, "<f4")]
    cols += [view(p, "<f4") for p in (v.vx_dev, v.vy_dev)] + ([view(v.vz_dev, "<f4")] if vz else [])
    rows = torch.empty((count, len(cols)), device="cuda")
    rows[pid.long()] = torch.stack(cols, 1)
    return rows[:loaded]


def _state_of(s):
    """The particles by id and the field energies of the pass's steps."""
    h, k, counts = s["handle"], s["case"]["steps"], s["counts"]
    fe = h.history(P.HIST_FIELD_ENERGY, s["at"] - k + 1, k)
    vz = s["case"]["kind"] == "mcc"
    now = h.diagnostics().n if vz else counts
    own, cur = torch.cuda.ExternalStream(h.stream()), torch.cuda.current_stream()
    cur.wait_stream(own)
    rows = [_by_id(h, i, now[i], n, vz) for i, n in enumerate(counts)]
    own.wait_stream(cur)
    if len(rows) == 3:
        # which neutrals of a cell pair up follows from their order in storage,
        # which differs from run to run: their positions alone can be compared
        rows[2] = rows[2][:, :2]
    return {"particles": rows, "field_energy": fe.astype(np.float32)}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "step":
        s["handle"].step(case["steps"])
        s["at"] += case["steps"]
        return _state_of(s)
    if kind == "staged":
        h = s["handle"]
        h.sort()
        for _ in range(case["steps"]):
            h.gather_push(True)
            h.poisson()
        s["at"] += case["steps"]
        return _state_of(s)
    if kind == "run_host":
        return s["handle"].run_host(*s["arrays"], case["steps"], prime=True, out=s["out"])
    if kind == "ensemble":
        e, k = s["ensemble"], case["steps"]
        e.step(k)
        s["at"] += k
        at, runs = s["at"], range(case["runs"])
        least = min(runs, key=lambda r: s["specs"][r].n)
        a = e.get_particles(least)
        out = {q: a[q].astype(np.float32) for q in a}
        # the sweep's result: every run's history of these steps (the kinetic
        # energy belongs to the push, one step earlier)
        for name, which, first in (("field_energy", P.HIST_FIELD_ENERGY, at - k + 1),
                                   ("kinetic_energy", P.HIST_KINETIC, at - k)):
            out[name] = np.stack([e.history(r, which, first, k) for r in runs]).astype(np.float32)
        return out
    if kind == "adjoint":
        for a in s["leaves"]:
            a.grad = None
        J = s["energy"](*s["leaves"])
        J.backward()
        return {"J": J.detach().float(), "grad": [a.grad for a in s["leaves"]]}
    if kind == "ensemble_adjoint":
        res, per = s["ensemble"].adjoint(s["specs"], case["steps"], case["every"])
        return {"J": np.array(res, np.float32), "grad": per}
    if kind == "compat_run":
        return P.compat_run(s["params"], *s["arrays"])[:2]
    return P.compat_run_steps(s["params"], *s["arrays"], case["steps"])


# ------------------------------------------------------------------ work
def work(case):
    """A step reads and writes every particle (cell, two offsets, two velocities: 20
    bytes) and every cell's density (8 bytes) and field (8) once each; per
    particle a four-node gather, push and deposit, per cell three transforms."""
    kind, k = case["kind"], case["steps"]

    def steps(particles, cells):
        return (k * (40.0 * particles + 32.0 * cells),
                k * (60.0 * particles + 15.0 * cells * math.log2(cells)))

    if kind in ("ensemble", "ensemble_adjoint"):
        per = [steps(side * side * ppc, side * side) for side, ppc, _, _ in _batch(case)]
        b, f = sum(p[0] for p in per), sum(p[1] for p in per)
        n = sum(side * side * ppc for side, ppc, _, _ in _batch(case))
    elif kind in ("compat_run", "compat_steps"):
        # 64-bit positions, velocities and forces in and out, density and field
        n, cells = case["npx"] * case["npy"], case["nx"] * case["ny"]
        return {"bytes": k * (96.0 * n + 64.0 * cells) + 48.0 * n,
                "flops": k * (150.0 * n + 15.0 * cells * math.log2(cells))}
    elif kind == "mcc":
        cells = case["nx"] * case["ny"]
        ne, nn = cells * case["electrons"], cells * case["neutrals"]
        b, f = steps(2 * ne + nn, cells)
        # an id and ten rounds of random numbers per electron, a cell list for the neutrals
        return {"bytes": b + k * (4.0 * ne + 8.0 * nn), "flops": f + k * 80.0 * ne}
    else:
        n = case["particles"]
        b, f = steps(n, case["nx"] * case["ny"])
        if kind == "run_host":
            b += 64.0 * n
    if kind in ("adjoint", "ensemble_adjoint"):
        # backwards: positions, adjoint state in and out for the kick, and for the gather
        b, f = b + k * 88.0 * n + 32.0 * n, 3.0 * f
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64 bits
def _cic(x, y, nx, ny):
    """Node indices and weights of positions in cells."""
    fx, fy = torch.floor(x.detach()), torch.floor(y.detach())
    cx, cy = fx.long() % nx, fy.long() % ny
    ax, ay = x - fx, y - fy
    x1, y1 = (cx + 1) % nx, (cy + 1) % ny
    return ((cy * nx + cx, (1 - ax) * (1 - ay)), (cy * nx + x1, ax * (1 - ay)),
            (y1 * nx + cx, (1 - ax) * ay), (y1 * nx + x1, ax * ay))


def _field(x, y, q, case):
    """Ex, Ey (flat) and the field energy of particles at x, y (cells)."""
    nx, ny = case["nx"], case["ny"]
    Lx, Ly, _ = _domain(case)
    dA = Lx / nx * Ly / ny
    rho = torch.zeros(nx * ny, dtype=torch.float64, device="cuda")
    for i, w in _cic(x, y, nx, ny):
        rho = rho.index_add(0, i, w * (q / dA))
    r = torch.fft.rfft2(rho.view(ny, nx))
    kx = TWO_PI / Lx * torch.arange(nx // 2 + 1, dtype=torch.float64, device="cuda")[None, :]
    ky = TWO_PI * torch.fft.fftfreq(ny, Ly / ny, dtype=torch.float64, device="cuda")[:, None]
    k2 = kx * kx + ky * ky
    k2[0, 0] = 1.0
    if nx % 2 == 0:
        kx[0, -1] = 0.0  # the derivative's Nyquist mode
    if ny % 2 == 0:
        ky[ny // 2, 0] = 0.0
    phi = r / k2
    phi = phi * (torch.arange(phi.numel(), device="cuda").view(phi.shape) > 0)
    ex = torch.fft.irfft2(-1j * kx * phi, s=(ny, nx)).reshape(-1)
    ey = torch.fft.irfft2(-1j * ky * phi, s=(ny, nx)).reshape(-1)
    return ex, ey, 0.5 * dA * (ex * ex + ey * ey).sum()


def _leapfrog(case, x, y, vx, vy):
    """The run from unprimed particles: final state (positions in cells) and energies."""
    nx, ny = case["nx"], case["ny"]
    Lx, Ly, dt = _domain(case)
    q = -Lx * Ly / case["particles"]
    x, y, energies = x * (nx / Lx), y * (ny / Ly), []

    def kick(vx, vy, ex, ey, c):
        fx = sum(w * ex[i] for i, w in _cic(x, y, nx, ny))
        fy = sum(w * ey[i] for i, w in _cic(x, y, nx, ny))
        return vx - c * fx, vy - c * fy

    ex, ey, _ = _field(x, y, q, case)
    vx, vy = kick(vx, vy, ex, ey, -0.5 * dt)
    for _ in range(case["steps"]):
        vx, vy = kick(vx, vy, ex, ey, dt)
        x, y = torch.remainder(x + vx * (dt * nx / Lx), nx), torch.remainder(y + vy * (dt * ny / Ly), ny)
        ex, ey, e = _field(x, y, q, case)
        energies.append(e)
    return x, y, vx, vy, energies


def _reference_run(case, seed):
    """The reference's step with its conventions (opposite-corner weights, ghost
    cells, k without the domain's length, swapped field axes, lagged kicks)."""
    p, arrays = _compat(case, seed)
    x, y, vx, vy = (torch.from_numpy(a).cuda() for a in arrays)
    nx, ny, Y, nyh = p.nx, p.ny, p.ny + 2, p.ny // 2 + 1
    dx, dy, dt, qm = p.xDim / nx, p.yDim / ny, p.dt, p.charge / p.mass
    i = torch.arange(nx, device="cuda")[:, None]
    j = torch.arange(nyh, device="cuda")[None, :]
    k1 = TWO_PI * torch.where(2 * i < nx, i, i - nx).double()
    k2 = TWO_PI * torch.where(2 * j < nyh, j, j - ny).double()
    k = k1 * k1 + k2 * k2
    k[0, 0] = math.inf
    grids = torch.zeros((4, nx + 2, Y), dtype=torch.float64, device="cuda")
    rho, phi, ex, ey = grids
    fox, foy = torch.zeros_like(x), torch.zeros_like(x)

    def cells():
        return (x / dx).long(), (y / dy).long()

    def weights():
        cx, cy = cells()
        a, b = x - cx * dx, y - cy * dy
        c, d = (cx * dx + dx) - x, (cy * dy + dy) - y
        A = dx * dy
        return cx, cy, (cx + 1) % nx, (cy + 1) % ny, (a * b / A, c * b / A, a * d / A, c * d / A)

    def ghosts(g, first):
        cols = slice(first, Y - first)
        g[0, cols], g[nx + 1, cols] = g[nx, cols].clone(), g[1, cols].clone()
        g[1:nx + 1, 0], g[1:nx + 1, Y - 1] = g[1:nx + 1, ny].clone(), g[1:nx + 1, 1].clone()

    for _ in range(case["steps"]):
        cx, cy, x1, y1, w = weights()
        rho.zero_()
        for (r, c), a in zip(((cx, cy), (x1, cy), (cx, y1), (x1, y1)), w):
            rho.view(-1).index_add_(0, (1 + r) * Y + 1 + c, a * p.charge)
        ghosts(rho, 0)
        o = torch.fft.rfft2(rho[1:nx + 1, 1:ny + 1]) / -k
        phi[1:nx + 1, 1:ny + 1] = torch.fft.irfft2(o, s=(nx, ny)) / (nx * ny)
        ghosts(phi, 1)
        ex[1:nx + 1, 1:ny + 1] = (phi[1:nx + 1, 0:ny] - phi[1:nx + 1, 2:ny + 2]) / (2 * dx)
        ey[1:nx + 1, 1:ny + 1] = (phi[0:nx, 1:ny + 1] - phi[2:nx + 2, 1:ny + 1]) / (2 * dy)
        at = [r * Y + c for r, c in ((cx, cy), (x1, cy), (cx, y1), (x1, y1))]
        fx = qm * sum(a * ex.view(-1)[n] for a, n in zip(w, at))
        fy = qm * sum(a * ey.view(-1)[n] for a, n in zip(w, at))
        vx, vy = vx + 0.5 * dt * fox, vy + 0.5 * dt * foy
        x, y = x + vx * dt, y + vy * dt
        x = torch.where(x > p.xDim, x - p.xDim, torch.where(x < 0, x + p.xDim, x))
        y = torch.where(y > p.yDim, y - p.yDim, torch.where(y < 0, y + p.yDim, y))
        vx, vy, fox, foy = vx + 0.5 * dt * fx, vy + 0.5 * dt * fy, fx, fy
    return dict(x=x, y=y, vx=vx, vy=vy, rho=rho, phi=phi, ex=ex, ey=ey)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("compat_run", "compat_steps"):
        if case["npx"] * case["npy"] * case["steps"] > EXACT_MAX:
            return None
        r = _reference_run(case, seed)
        return (r["x"], r["y"]) if kind == "compat_run" else r
    if kind not in ("staged", "step", "run_host", "adjoint"):
        return None  # random collisions, loads by the library's own generator
    n = case["particles"]
    if n * case["steps"] > EXACT_MAX or (kind in ("staged", "step") and n > HOST_LOAD_MAX):
        return None
    Lx, Ly, _ = _domain(case)
    start = _plasma(case, seed)
    if kind == "adjoint":
        if n * case["steps"] > EXACT_MAX // 16:
            return None  # every step's intermediates are kept
        leaves = [a.requires_grad_() for a in start]
        J = _leapfrog(case, *leaves)[4][-1]
        J.backward()
        return {"J": J.detach(), "grad": [a.grad for a in leaves]}
    x, y, vx, vy, energies = _leapfrog(case, *start)
    if kind == "run_host":
        return [a.cpu().numpy() for a in (x * (Lx / case["nx"]), y * (Ly / case["ny"]), vx, vy)]
    return {"particles": [torch.stack([x, y, vx, vy], 1)], "field_energy": torch.stack(energies)}
