"""The reference-convention path's division by known divisors (div_known.cu)
gives the general division's result: on random operands, next to exact
quotients and to midpoints, for zeros and near the ends of its range."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

import build_lib

pytestmark = pytest.mark.gpu

# cell sizes, areas, 2 dx and -k^2 of the path's grids, and divisors whose
# mantissas are next to 1 and 2, where the product is furthest off
DIVISORS = ([10 / 32, 10 / 128, 7 / 12, 12 / 1024, 13 / 192, 1 / 3, (10 / 32) * (10 / 31), 2 * (7 / 9)] +
            [-((2 * math.pi * i) ** 2 + (2 * math.pi * j) ** 2) for i, j in ((0, 1), (3, 5), (96, 96), (511, 512))] +
            [math.nextafter(1.0, 2.0), math.nextafter(2.0, 1.0), 1.0 + 3 * 2.0 ** -52, 2.0 - 5 * 2.0 ** -52, 1.0, -0.75])


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("div") / "div_known.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "div_known.cu")
    subprocess.run([build_lib.NVCC] + build_lib.COMMON + ["--fmad=false", "-shared", src, "-o", so], check=True)
    lib = C.CDLL(so)
    lib.div_given.restype = lib.div_drawn.restype = C.c_longlong
    return lib


@pytest.mark.parametrize("b", DIVISORS)
def test_random_operands(lib, b):
    # the path's range, and nearly all of the format's
    for seed, lo, hi, n in ((1, 60, 60, 1 << 27), (2, 870, 870, 1 << 24)):
        assert lib.div_drawn(C.c_ulonglong(seed), C.c_longlong(n), lo, hi, C.c_double(b)) == 0


@pytest.mark.parametrize("b", DIVISORS)
def test_edges(lib, b):
    rng = np.random.default_rng(int(abs(b) * 1e6) % 2 ** 31)
    with np.errstate(all="ignore"):
        q = np.concatenate([np.arange(1.0, 2000.0), rng.integers(1, 1 << 53, 200_000).astype(float),
                            rng.random(200_000)])
        near = [q * b]  # products that round, and their neighbours on both sides
        for toward in (np.inf, -np.inf):
            x = q * b
            for _ in range(3):
                x = np.nextafter(x, toward)
                near.append(x)
        # halfway between two quotients: (q + ulp / 2) b
        near += [(q + 0.5 * np.spacing(q)) * b, np.nextafter(q, np.inf) * b]
        ends = np.array([0.0, -0.0] + [t * 2.0 ** e for t in (1.0, -1.5) for e in (-870, 870)])
        a = np.ascontiguousarray(np.concatenate(near + [ends]))
    assert lib.div_given(a.ctypes.data_as(C.c_void_p), C.c_longlong(len(a)), C.c_double(b)) == 0
