"""Reference-convention GPU path (pic_compat_run*, the picFloatGpu drop-in)
against the reference's own CPU step: golden vectors made from the
reference's sources, and the bit-exact C restatement for other inputs."""
import glob
import os

import numpy as np
import pytest

import oracle as O
import picgpu as P
from conftest import GOLDEN

pytestmark = pytest.mark.gpu
CASES = sorted(glob.glob(os.path.join(GOLDEN, "compat_*.npz")))
INTS = {"xDim", "yDim", "nx", "ny", "npx", "npy"}


def case(path):
    z = np.load(path)
    d = {str(k): (int(v) if str(k) in INTS else float(v)) for k, v in zip(z["param_keys"], z["params"])}
    return P.ref_params(**d), z


@pytest.mark.parametrize("path", CASES, ids=[os.path.basename(c) for c in CASES])
def test_compat_steps_match_reference(path):
    p, z = case(path)
    out = P.compat_run_steps(p, z["x0"], z["y0"], z["vx0"], z["vy0"], int(z["nsteps"]))
    # FP64 throughout; the GPU sums the deposit with atomics and transforms with
    # cuFFT, so agreement is to rounding, far inside the reference's own 1e-4
    # position check (collisionless/double/src/main.cc:260)
    for k in ("x", "y", "vx", "vy"):
        np.testing.assert_allclose(out[k], z[k], rtol=0, atol=1e-9, err_msg=k)
    for k in ("rho", "phi", "ex", "ey"):
        scale = max(np.abs(z[k]).max(), 1e-300)
        np.testing.assert_allclose(out[k], z[k], rtol=0, atol=1e-10 * scale, err_msg=k)


@pytest.mark.parametrize("path", CASES, ids=[os.path.basename(c) for c in CASES])
def test_compat_run_counts_steps_like_reference(path):
    p, z = case(path)
    xo, yo, sec = P.compat_run(p, z["x0"], z["y0"], z["vx0"], z["vy0"])
    ref = P.compat_run_steps(p, z["x0"], z["y0"], z["vx0"], z["vy0"], int(z["loop_steps"]))
    # two GPU runs agree to the last bits only: the FP64 deposit atomics sum
    # in scheduling order; one step more or less would move particles by
    # v dt, orders of magnitude above this tolerance
    np.testing.assert_allclose(xo, ref["x"], rtol=0, atol=1e-9)
    np.testing.assert_allclose(yo, ref["y"], rtol=0, atol=1e-9)
    assert sec > 0


def test_compat_larger_case_vs_restatement():
    p = O.ref_params(xDim=16, yDim=16, nx=64, ny=64, npx=200, npy=150, dt=0.005, tmax=1.0,
                     charge=-20.0, mass=5.0, vtx=1.0, vty=1.0, vdx=0.5, vdy=0.0)
    x, y, vx, vy = O.compat_init(p, seed=11)
    ref = O.compat_run(p, x, y, vx, vy, 30, nthreads=0)
    out = P.compat_run_steps(P.ref_params(**{f[0]: getattr(p, f[0]) for f in p._fields_}),
                             x, y, vx, vy, 30)
    for k in ("x", "y", "vx", "vy"):
        np.testing.assert_allclose(out[k], ref[k], rtol=0, atol=1e-9, err_msg=k)


@pytest.mark.parametrize("nx,ny", [(8, 8), (8, 1024), (1024, 8), (16, 64), (64, 32), (128, 16),
                                   (12, 10), (2, 3), (16, 20), (9, 32)])
def test_compat_grid_sizes_vs_restatement(nx, ny):
    """The own power-of-two transforms (one and several per block, with and
    without a radix-2 pass) and the cuFFT path, from particles in the domain,
    on its edges and slightly outside it."""
    rng = np.random.default_rng(nx * 1000 + ny)
    kw = dict(xDim=7, yDim=12, nx=nx, ny=ny, npx=37, npy=11, dt=0.01, tmax=1.0, charge=-30.0,
              mass=7.0)
    n = 37 * 11
    x, y = rng.uniform(0, 7, n), rng.uniform(0, 12, n)
    x[:6] = [0.0, 7.0, -0.0, 7.0 / nx, -0.01 / nx, 7.0]
    y[:6] = [12.0, 0.0, 12.0, 12.0 / ny, 12.0, -0.01 / ny]
    vx, vy = rng.normal(0, 3.0, n), rng.normal(0, 3.0, n)
    ref = O.compat_run(O.ref_params(**kw), x, y, vx, vy, 12)
    out = P.compat_run_steps(P.ref_params(**kw), x, y, vx, vy, 12)
    # FP64 with another summation and transform order: the bounds of the
    # golden cases above
    for k in ("x", "y", "vx", "vy"):
        np.testing.assert_allclose(out[k], ref[k], rtol=0, atol=1e-9, err_msg=k)
    for k in ("rho", "phi", "ex", "ey"):
        scale = max(np.abs(ref[k]).max(), 1e-300)
        np.testing.assert_allclose(out[k], ref[k], rtol=0, atol=1e-10 * scale, err_msg=k)


@pytest.mark.parametrize("nx,ny", [(64, 64), (30, 20)])
def test_short_memory_computes_the_weights_again(nx, ny, monkeypatch):
    """Within PIC_STAGE_MAX_BYTES a run holds no weights per particle (at most 64
    bytes each instead of 88) and agrees to the order of the deposit's sums."""
    import threading

    import torch

    kw = dict(xDim=10, yDim=10, nx=nx, ny=ny, npx=2000, npy=1500, dt=0.01, tmax=1.0)
    n = 3_000_000
    rng = np.random.default_rng(nx)
    state = [rng.uniform(0, 10, n), rng.uniform(0, 10, n), rng.normal(0, 1, n), rng.normal(0, 1, n)]

    def go():
        torch.cuda.synchronize()
        free, least, stop = torch.cuda.mem_get_info()[0], [1 << 60], threading.Event()

        def watch():
            while not stop.is_set():
                least[0] = min(least[0], torch.cuda.mem_get_info()[0])

        t = threading.Thread(target=watch)
        t.start()
        out = P.compat_run_steps(P.ref_params(**kw), *state, 20)
        stop.set()
        t.join()
        return out, free - least[0]

    go()  # libraries loaded
    ref, _ = go()
    monkeypatch.setenv("PIC_STAGE_MAX_BYTES", str(1 << 20))
    out, used = go()
    print("bytes per particle", used / n)
    assert used < 64 * n + (24 << 20)
    for k in ("x", "y", "vx", "vy"):
        np.testing.assert_allclose(out[k], ref[k], rtol=0, atol=1e-9, err_msg=k)
