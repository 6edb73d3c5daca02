"""The step's launch rules change how the work is split, not its results: the
deposit is an integer sum and a particle's push does not depend on its block,
so the particles and the density agree bit for bit."""
import numpy as np
import pytest

import picgpu as P

pytestmark = pytest.mark.gpu

NX, L, DT = 64, 4 * np.pi, 0.1


def load(n, seed):
    rng = np.random.default_rng(seed)
    vx = np.where(np.arange(n) % 2 == 0, 0.2, -0.2) + 0.01 * rng.normal(size=n)
    return rng.random(n) * L, rng.random(n) * L, vx, 0.3 * rng.normal(size=n)


def run(parts, steps, **tuning):
    """One species per part of the load, all of one charge and mass."""
    total = sum(len(p[0]) for p in parts)
    w = L * L / total
    h = P.Handle(P.config(NX, NX, L, L, DT, [P.species(len(p[0]), -w, w, -1) for p in parts], **tuning))
    with h:
        for s, p in enumerate(parts):
            h.set_particles(s, *p)
        h.prime_leapfrog()
        h.step(steps)
        got = [h.get_particles(s) for s in range(len(parts))]
        d = h.diagnostics()
        rho = h.rho_fixed()
    assert d.error_flags == 0 and d.total_charge_fixed == d.expected_charge_fixed
    return {k: np.concatenate([g[k] for g in got]) for k in ("x", "y", "vx", "vy")}, rho


def same(a, b):
    for k in a[0]:
        np.testing.assert_array_equal(a[0][k], b[0][k], err_msg=k)
    np.testing.assert_array_equal(a[1], b[1])


@pytest.mark.parametrize("n", [1, 1023, 1025, 152 * 4 * 1024 - 1, 152 * 4 * 1024 + 1, 1_500_003])
def test_default_chunk_matches_given_chunks(n):
    """Push blocks sized from the particle count, below and above one wave of
    blocks on the GPU, with a last block of any length; through a sort."""
    p = [load(n, n)]
    auto = run(p, 7, sort_every=3)
    for chunk in (1024, 4096):
        same(auto, run(p, 7, sort_every=3, chunk=chunk))


@pytest.mark.parametrize("split", [(0.5, 0.5), (0.9, 0.1), (0.4, 0.35, 0.25)])
def test_species_pushed_side_by_side_match_one_species(split):
    """Two or three species whose pushes overlap against one species of all
    their particles."""
    n = 300_001
    p = load(n, 3)
    cut = [0] + [int(round(n * c)) for c in np.cumsum(split)]
    cut[-1] = n
    parts = [tuple(a[i:j] for a in p) for i, j in zip(cut, cut[1:])]
    same(run([p], 25, sort_every=10), run(parts, 25, sort_every=10))


def test_a_reload_with_another_count_steps_as_a_fresh_handle():
    """The background that the solve subtracts follows the loaded count: a
    handle with a given push chunk, stepped, loaded with more particles and
    stepped again, against a handle loaded with them at once."""
    first, then = load(NX * NX * 16, 5), load(NX * NX * 20, 6)
    n = len(then[0])
    cfg = P.config(NX, NX, L, L, DT, [P.species(n, -L * L / n, L * L / n, -1)], chunk=1024, sort_every=3)
    got = []
    for loads in ((first, then), (then,)):
        with P.Handle(cfg) as h:
            for a in loads:
                h.set_particles(0, *a)
                h.prime_leapfrog()
                h.step(7)
            got.append((h.get_particles(0), h.grid(P.GRID_RHO)))
    same(*got)


@pytest.mark.parametrize("before", ["deposit", "gather_push"])
def test_steps_after_a_deposit_without_a_solve(before):
    """A density that was deposited and never solved for is not counted twice
    by the step that follows."""
    n = NX * NX * 16
    w = L * L / n
    with P.Handle(P.config(NX, NX, L, L, DT, [P.species(n, -w, w, -1)])) as h:
        h.set_particles(0, *load(n, 8))
        h.prime_leapfrog()
        getattr(h, before)()
        h.step(1)
        d = h.diagnostics()
        assert d.error_flags == 0 and d.total_charge_fixed == d.expected_charge_fixed
        if before == "deposit":
            got = h.get_particles(0), h.rho_fixed()
            h.set_particles(0, *load(n, 8))
            h.prime_leapfrog()
            h.step(1)
            same(got, (h.get_particles(0), h.rho_fixed()))


def test_a_mostly_empty_handle_steps_as_fast_as_a_full_one():
    """A step's cost follows the particles, not the room for them: 16 per cell
    on 64^2 in a handle for 64 M (which took six times as long with a block
    for every 1024 slots; the bound leaves a factor of two for noise)."""
    import torch

    n = NX * NX * 16
    w = L * L / n
    best, got = [], []
    for cap in (n, 1 << 26):
        with P.Handle(P.config(NX, NX, L, L, DT, [P.species(cap, -w, w, -1)], sort_every=200)) as h:
            h.set_particles(0, *load(n, 9))
            h.prime_leapfrog()
            h.step(1)
            st = torch.cuda.ExternalStream(h.stream())
            times = []
            for _ in range(5):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record(st)
                h.step(30)
                b.record(st)
                h.synchronize()
                times.append(a.elapsed_time(b))
            best.append(min(times))
            got.append((h.get_particles(0), h.rho_fixed()))
    print("ms for 30 steps", best)
    same(*got)
    assert best[1] < 2.0 * best[0]


@pytest.mark.parametrize("nx,ny,ppc", [(512, 512, 64), (700, 640, 32), (1024, 512, 26)])
def test_default_blocks_of_large_runs_hold_their_tile(nx, ny, ppc):
    """From about two waves of blocks on the default is the layout of a chunk of
    8192 (a few per cent faster there than whole waves of another size): the
    same storage order after a sort."""
    n = nx * ny * ppc + 3
    w = L * L / n
    order = []
    for chunk in (0, 8192):
        with P.Handle(P.config(nx, ny, L, L, DT, [P.species(n, -w, w, -1)], chunk=chunk)) as h:
            h.init_particles(0, P.init_spec(n, vth=(0.1, 0.1, 0.0), seed=4))
            order.append(h.get_particles_raw(0)["cell"])
    np.testing.assert_array_equal(*order)


def test_handles_of_two_threads_launch_with_windows_of_different_size():
    """One handle per host thread: pushes whose windows take 52 and 85 KB of
    shared memory, launched one by one from two threads at a time."""
    import threading

    n = NX * NX * 16
    w = L * L / n
    p = load(n, 12)
    results, errors = {}, []

    def work(halo, steps):
        try:
            with P.Handle(P.config(NX, NX, L, L, DT, [P.species(n, -w, w, -1)], chunk=4096, tile_w=16, tile_h=16,
                                   halo=halo)) as h:
                h.set_particles(0, *p)
                h.prime_leapfrog()
                for _ in range(steps):
                    h.gather_push(True)
                    h.poisson()
                results[halo, steps] = h.get_particles(0), h.rho_fixed()
        except P.PicError as e:
            errors.append(e)

    for halo in (10, 16):
        work(halo, 1500)
    alone = dict(results)
    for _ in range(3):
        threads = [threading.Thread(target=work, args=(halo, 1500)) for halo in (10, 16, 10, 16)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors[0]
        for k in alone:
            same(results[k], alone[k])
