"""The fixed-point pair functions (pair_fixed.cuh) on the host, coefficient by coefficient against
extended precision."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
U = 2.0**-53


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = tmp_path_factory.mktemp("pair_fixed") / "pair_fixed.so"
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "host" / "pair_fixed_host.cpp")], check=True)
    L = ctypes.CDLL(str(so))
    D = ctypes.c_double
    L.wall_block.argtypes = [D] * 5 + [ctypes.c_void_p]
    L.radial_block.argtypes = [ctypes.c_int] + [D] * 5 + [ctypes.c_void_p]
    return L


def call(fn, n, *args):
    out = np.empty(n)
    fn(*args, out.ctypes.data)
    return out


def wall_reference(x, y, t, h, e):
    """2 t h times the free Stokeslet and the images over d_j d_k, d_j, 1 (pair_math.cuh's header), and the size of
    the terms of b1 and b2."""
    x, y, t, h, e = (np.longdouble(v) for v in (x, y, t, h, e))
    dm, dp = t - h, t + h
    rq = x * x + y * y + e * e
    sF, s = 1 / np.sqrt(rq + dm * dm), 1 / np.sqrt(rq + dp * dp)
    Z1 = 2 * sF**2 * s**2 / (sF + s)
    Z3 = Z1 * (sF**2 + sF * s + s**2)
    k = 2 * t * h
    p, r = Z3, 3 * s**5
    return k * (p + r), k * (p * dm - r * dp), k * (p * dm + r * dp), k * (abs(p * dm) + abs(r * dp))


@pytest.mark.parametrize("height", [1.0, 1e-3, 1e-6, 1e-9, 1e-12])
def test_wall_coefficients_between_height_and_plane(lib, height):
    """xz and zx entries are products of the displacement along the wall and a coefficient that shrinks with the
    heights: its error stays a few roundings of its own terms, whatever the heights are beside the distance."""
    rng = np.random.default_rng(1)
    for _ in range(400):
        x, y = rng.uniform(-1, 1, 2)
        t, h = height * rng.uniform(0.1, 1.0, 2)
        e = 10.0 ** rng.uniform(-4, -1)
        a, b1, b2, _, _ = call(lib.wall_block, 5, x, y, t, h, e)
        ra, rb1, rb2, size = wall_reference(x, y, t, h, e)
        # squared distances, two roots, the coefficients and two products: a dozen roundings
        assert abs(a - ra) <= 12 * U * abs(ra)
        assert abs(b1 - rb1) <= 12 * U * size
        assert abs(b2 - rb2) <= 12 * U * size


@pytest.mark.parametrize("gap", [1.0, 1e-4, 1e-8])
def test_wall_coefficients_far_from_the_wall(lib, gap):
    """Source and target close to one another and far above the wall, at nearly the same height."""
    rng = np.random.default_rng(2)
    for _ in range(400):
        x, y = gap * rng.uniform(-1, 1, 2)
        h = rng.uniform(1.0, 30.0)
        t = h * (1 + gap * rng.uniform(-1e-3, 1e-3))
        e = gap * 10.0 ** rng.uniform(-3, 0)
        a, b1, b2, _, _ = call(lib.wall_block, 5, x, y, t, h, e)
        ra, rb1, rb2, size = wall_reference(x, y, t, h, e)
        assert abs(a - ra) <= 12 * U * abs(ra)
        assert abs(b1 - rb1) <= 12 * U * size
        assert abs(b2 - rb2) <= 12 * U * size
