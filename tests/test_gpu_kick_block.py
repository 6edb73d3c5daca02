"""The adjoint's scatter windows on their own (kick_block.cu): fixed-point sums
against FP64 and FP32 ones, for adjoint velocities of one size, of sizes that
vary over the grid, and with a few far above the rest."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import build_lib

pytestmark = pytest.mark.gpu

NX = NY = 64
TW, TH, HALO, CHUNK = 16, 16, 3, 8192


@pytest.fixture(scope="module")
def kick(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("kick") / "kick_block.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "kick_block.cu")
    subprocess.run([build_lib.NVCC] + build_lib.COMMON + ["-shared", src, "-o", so], check=True)
    lib = C.CDLL(so)

    def run(cell, ox, oy, avx, avy):
        n = len(cell)
        first = cell[::CHUNK]
        anchor = ((first & 0xFFFF) // TW | ((first >> 16) // TH) << 16).astype(np.int32)
        g = np.empty((2, NX * NY), np.float32)
        args = [np.ascontiguousarray(a).ctypes.data_as(C.c_void_p) for a in (anchor, cell, ox, oy, avx, avy, g[0], g[1])]
        assert lib.kick_scatter(NX, NY, TW, TH, HALO, C.c_longlong(n), CHUNK, *args[:6],
                                g[0].ctypes.data_as(C.c_void_p), g[1].ctypes.data_as(C.c_void_p)) == 0
        return g

    return run


def load(ppc, seed):
    """Particles in tile order, some of them drifted out of their block's window."""
    rng = np.random.default_rng(seed)
    n = NX * NY * ppc
    cx, cy = rng.integers(0, NX, n), rng.integers(0, NY, n)
    o = np.lexsort((cx, cy, cx // TW, cy // TH))
    cx, cy = cx[o], cy[o]
    far = rng.random(n) < 0.01
    cx = np.where(far, (cx + rng.integers(0, NX, n)) % NX, cx)
    off = rng.random((2, n)).astype(np.float32)
    return (cx | cy << 16).astype(np.int32), off[0], off[1], rng


def sums(cell, ox, oy, v):
    """sum w v per node in FP64 and in FP32, one after the other, and sum w |v|."""
    cx, cy = cell & 0xFFFF, cell >> 16
    gx, gy = np.float32(1) - ox, np.float32(1) - oy
    s, a, f = np.zeros(NX * NY), np.zeros(NX * NY), np.zeros(NX * NY, np.float32)
    for w, i, j in ((gx * gy, 0, 0), (ox * gy, 1, 0), (gx * oy, 0, 1), (ox * oy, 1, 1)):
        node = (cy + j) % NY * NX + (cx + i) % NX
        p = w.astype(np.float64) * v.astype(np.float64)
        s += np.bincount(node, p, NX * NY)
        a += np.bincount(node, np.abs(p), NX * NY)
        np.add.at(f, node, w * v)
    return s, f, a


@pytest.mark.parametrize("kind", ["one size", "a wave", "outlier 2^12", "outlier 2^30", "outliers 0.1 %", "zeros"])
@pytest.mark.parametrize("ppc", [16, 64])
def test_scatter_no_further_off_than_float_sums(kick, kind, ppc):
    """Each node's error, relative to the sum of its contributions' sizes: over
    the grid it is no larger than that of the same sums in FP32 (half as much
    again allowed for their order), beside values far above the rest too."""
    cell, ox, oy, rng = load(ppc, ppc)
    n = len(cell)
    v = rng.normal(size=(2, n))
    if kind == "a wave":
        v *= np.sin(2 * np.pi * ((cell & 0xFFFF) + ox) / NX)
    elif kind == "outliers 0.1 %":
        v[:, rng.random(n) < 1e-3] *= 2.0 ** rng.integers(8, 24)
    elif kind == "zeros":
        v[:, rng.random(n) < 0.9] = 0.0
    elif kind != "one size":
        v[:, n // 2] = 2.0 ** int(kind.split("^")[1])
    v = v.astype(np.float32)
    g = kick(cell, ox, oy, v[0], v[1])
    for k in range(2):
        s, f, a = sums(cell, ox, oy, v[k])
        on = a > 0
        here, plain = (np.sqrt(np.mean(((x - s)[on] / a[on]) ** 2)) for x in (g[k], f))
        print(f"{kind} {ppc}: rms error {here:.2e}, of FP32 sums {plain:.2e}")
        assert here < 1.5 * plain
