"""pic_run_host, the one-call run from and to host memory (how the
reference's picFloatGpu is used, thesisCode/collisionless/double/src/
main.cc:182): the same state as the staged calls, outputs that alias the
inputs, page-locked or pageable arrays, and the FP64 oracle over a short
run from the imported state."""
import numpy as np
import pytest
import torch

import oracle as O
import picgpu as P
from gpu_util import normalized_electrons, periodic_diff

pytestmark = pytest.mark.gpu

NX = NY = 64
L = 4 * np.pi
DT = 0.1
STEPS = 30


def _load(n, seed=21):
    rng = np.random.default_rng(seed)
    x = rng.random(n) * L
    x = (x + 0.05 * np.sin(2 * np.pi * x / L)) % L  # a density wave on mode 1
    y = rng.random(n) * L
    vx = rng.normal(0.0, 0.05, n) + np.where(np.arange(n) % 2 == 0, 0.2, -0.2)
    vy = rng.normal(0.0, 0.05, n)
    return x, y, vx, vy


def test_run_host_matches_staged_calls_and_fp64_oracle():
    n = NX * NY * 16
    cfg, q, m = normalized_electrons(NX, NY, L, L, n, DT)
    arrs = _load(n)
    with P.Handle(cfg) as h:
        out = h.run_host(*arrs, STEPS)
        d = h.diagnostics()
        assert d.error_flags == 0 and d.step == STEPS
        assert d.total_charge_fixed == d.expected_charge_fixed
    with P.Handle(cfg) as h:
        h.set_particles(0, *arrs)
        start = h.get_particles()
        h.prime_leapfrog()
        h.step(STEPS)
        staged = h.get_particles()
    for k, o in zip(("x", "y", "vx", "vy"), out):
        np.testing.assert_array_equal(o, staged[k], err_msg=k)

    st = O.PhysState(NX, NY, L, L, DT, 1.0)
    st.add_species(start["x"], start["y"], start["vx"], start["vy"], q, m)
    st.prime(nthreads=0)
    st.run(STEPS, nthreads=0)
    s = st.species[0]
    cell = L / NX
    dxp = periodic_diff(out[0], s["x"], L)
    dyp = periodic_diff(out[1], s["y"], L)
    print("position max abs err (cells)", np.abs(dxp).max() / cell, np.abs(dyp).max() / cell)
    assert np.abs(dxp).max() < 1e-3 * cell
    assert np.abs(dyp).max() < 1e-3 * cell
    np.testing.assert_allclose(out[2], s["vx"], atol=1e-4 * np.abs(s["vx"]).max())
    np.testing.assert_allclose(out[3], s["vy"], atol=1e-4 * np.abs(s["vy"]).max())


def test_run_host_in_place_from_page_locked_arrays():
    n = NX * NY * 8 + 1
    cfg, _, _ = normalized_electrons(NX, NY, L, L, n, DT)
    arrs = _load(n, seed=22)
    with P.Handle(cfg) as h:
        ref = h.run_host(*arrs, 7, prime=False)
    pinned = [torch.from_numpy(a.copy()).pin_memory() for a in arrs]
    views = [t.numpy() for t in pinned]
    with P.Handle(cfg) as h:
        h.run_host(*views, 7, prime=False, out=views)
    for k in range(4):
        np.testing.assert_array_equal(views[k], ref[k])
    assert not np.array_equal(views[0], arrs[0])  # the particles moved


def test_run_host_rejects_more_particles_than_capacity():
    n = 1000
    cfg, _, _ = normalized_electrons(16, 16, 1.0, 1.0, n, DT)
    x, y, vx, vy = (np.zeros(n + 1) for _ in range(4))
    with P.Handle(cfg) as h:
        with pytest.raises(P.PicError):
            h.run_host(x, y, vx, vy, 1)


def test_run_host_keeps_the_library_transforms(monkeypatch):
    """On sides with factors 2, 3 and 5 the one-call run solves through the
    library, as PIC_FIELD_SOLVER=cufft does everywhere, while plain steps do
    not: the same bits before and after steps on the same handle, whose two
    sets of graphs stay apart."""
    nx, ny, n = 54, 45, 54 * 45 * 20 + 3
    cfg, _, _ = normalized_electrons(nx, ny, L, L, n, DT)
    arrs = _load(n, seed=23)

    def stepped(h):
        h.set_particles(0, *arrs)
        h.prime_leapfrog()
        h.step(25)
        return h.get_particles()

    with P.Handle(cfg) as h:
        first = h.run_host(*[a.copy() for a in arrs], 25)
        plain = stepped(h)
        again = h.run_host(*[a.copy() for a in arrs], 25)
        assert h.diagnostics().error_flags == 0
    monkeypatch.setenv("PIC_FIELD_SOLVER", "cufft")
    with P.Handle(cfg) as h:
        lib = h.run_host(*[a.copy() for a in arrs], 25)
        lib_stepped = stepped(h)
    for k, a, b, c in zip(("x", "y", "vx", "vy"), first, again, lib):
        np.testing.assert_array_equal(a, b, err_msg=k)
        np.testing.assert_array_equal(a, c, err_msg=k)
        np.testing.assert_array_equal(a, lib_stepped[k], err_msg=k)
        # rounding of the fields over 25 steps, as in test_gpu_spectral.py
        d = periodic_diff(plain[k], a, L) if k in "xy" else plain[k] - a
        assert np.abs(d).max() < 1e-4
    assert not np.array_equal(plain["vx"], first[2])


def test_adjoint_keeps_the_library_transforms(monkeypatch):
    """Likewise for the adjoint's forward steps, from its first field on: the
    final state and J to the last bit, the gradients to the order of their
    float sums."""
    nx, ny, n = 54, 45, 54 * 45 * 20 + 3
    cfg, _, _ = normalized_electrons(nx, ny, L, L, n, DT)
    arrs = _load(n, seed=24)
    got = []
    for solver in ("spectral", "cufft"):
        monkeypatch.setenv("PIC_FIELD_SOLVER", solver)
        with P.Handle(cfg) as h:
            h.set_particles(0, *arrs)
            r, *g = h.adjoint(20, every=6)
            got.append((r.J, g, h.get_particles(), h.history(P.HIST_FIELD_ENERGY, 0, 21)))
    (Ja, ga, pa, fa), (Jb, gb, pb, fb) = got
    assert Ja == Jb
    np.testing.assert_array_equal(fa, fb)
    for k in pa:
        np.testing.assert_array_equal(pa[k], pb[k], err_msg=k)
    for a, b in zip(ga, gb):
        assert np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("call", ["run_host", "one segment", "segments"])
def test_steps_after_a_library_solve_resume_bit_for_bit(call, tmp_path):
    """On sides with factors 2, 3 and 5 the field that the one-call run and the
    adjoint leave is a function of the particles alone, as after every other
    call: steps go on as from a state file of them."""
    nx, ny, n = 54, 45, 54 * 45 * 20 + 3
    cfg, _, _ = normalized_electrons(nx, ny, L, L, n, DT)
    arrs = _load(n, seed=25)
    path = str(tmp_path / "run.picstate")
    with P.Handle(cfg) as h:
        if call == "run_host":
            h.run_host(*[a.copy() for a in arrs], 20)
        else:
            h.set_particles(0, *arrs)
            h.adjoint(20, every=20 if call == "one segment" else 6)
        kept = h.history(P.HIST_FIELD_ENERGY, 0, 21)
        h.save(path)
        h.step(15)
        a, d, fa = h.get_particles(), h.diagnostics(), h.history(P.HIST_FIELD_ENERGY, 0, 36)
    with P.Handle(cfg) as h:
        h.load(path)
        h.step(15)
        b, fb = h.get_particles(), h.history(P.HIST_FIELD_ENERGY, 21, 15)
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    np.testing.assert_array_equal(fa[:21], kept)
    np.testing.assert_array_equal(fa[21:], fb)
    assert d.step == 35 and d.error_flags == 0 and d.total_charge_fixed == d.expected_charge_fixed
